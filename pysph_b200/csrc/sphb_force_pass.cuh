// sphb_force_pass.cuh -- the force pass, templated on the smoothing kernel.
// Included by one translation unit per kernel type (sphb_pass_*.cu), which
// instantiates launch_force_kt for its kernel and dimensions.
//
// MomentumEquation.eval_nbr (S/sph/funcs/pressure_funcs.pyx:246-391; OpenCL
// pressure_funcs.clt:69-157), per neighbour b of dest a:
//   dot = v_ab . r_ab,  dt_fac_a = max |h_ab dot / (r_ab^2 + eta^2 h_ab^2)|
//   tmp = P_a/rho_a^2 + P_b/rho_b^2 (+ Pi_ab when dot < 0,
//         Pi_ab = (-alpha c_ab mu + beta mu^2) / rho_ab, mu = h_ab dot /
//         (r_ab^2 + eta^2 h_ab^2))
//   a_a += -m_b tmp grad W(r_ab, h_ab)
// SPHPressureGradient (:62-161) is the same without Pi and dt_fac.
// GravityForce (S/sph/funcs/external_force.pyx:13-62) adds g afterwards.
// Per scene the kernel also keeps max dt_fac and max |a|^2 for the CFL rule.
// Variable h (scene.variable_h): the symmetric neighbour set r < radius_scale
// max(h_a, h_b); with scene.hks every pair function's W and grad W are the
// means of their values at h_a and h_b (pressure_funcs.pyx:141-149,
// 371-381), the viscosity and dt_fac keep h_ab.

#pragma once

#include <type_traits>

#include "sphb_kernels.cuh"
#include "sphb_launch.cuh"
#include "sphb_pairs.cuh"
#include "sphb_stage.cuh"

namespace sphb {

// Everything after the pair sums of dest k: its outputs (non-LocalReal
// dests get 0), gravity, dt_fac, the per-scene CFL maxima, the integrator
// stage fused into the epilogue and the pair count.  Every thread
// of the block calls it (block reductions inside); acc, dtf, drho and xs
// are valid in lane 0 of each dest; visc: the pass has a viscous term
// and writes dt_fac.
template <int DIM, bool F32, bool CONT>
__device__ __forceinline__ void force_finish(const sphb_engine &e, int cur, int k, int s, int a,
                                             bool active, int lane, double *acc, double dtf,
                                             double drho, const double *xs, bool visc,
                                             uint32_t mm, uint32_t rm, uint32_t xm,
                                             int with_gravity, int mode, unsigned int np)
{
    const sphb_scene &sc = e.scene[s];
    double a2 = 0.0, dtf_out = 0.0;
    if (CONT && active && lane == 0) {
        // non-LocalReal dests get 0 (S/sph/sph_func.pyx:220-227)
        const bool real = e.buf[cur].tag[k] == 0;
        if (rm) {
            const double v = real ? drho : 0.0;
            if (F32) ((float *)e.f.drho)[k] = (float)v;
            else ((double *)e.f.drho)[k] = v;
            if (!isfinite(v)) flag(e, SPHB_ST_NONFINITE_RHO);
        }
        if (xm) {
            void *xo[3] = {e.f.xu, e.f.xv, e.f.xw};
            for (int d = 0; d < DIM; ++d) {
                const double v = real ? xs[d] : 0.0;
                if (F32) ((float *)xo[d])[k] = (float)v;
                else ((double *)xo[d])[k] = v;
            }
        }
    }
    if (active && lane == 0 && mm) {
        const bool real = e.buf[cur].tag[k] == 0;
        if (real) {
            if (with_gravity) {
                acc[0] += sc.g[0];
                acc[1] += sc.g[1];
                if (DIM == 3) acc[2] += sc.g[2];
            }
            dtf_out = visc ? dtf : 0.0;
        } else {
            acc[0] = acc[1] = acc[2] = 0.0;
        }
        if (F32) {
            const float fx = (float)acc[0], fy = (float)acc[1], fz = (float)acc[2];
            ((float *)e.f.au)[k] = fx;
            ((float *)e.f.av)[k] = fy;
            if (DIM == 3) ((float *)e.f.aw)[k] = fz;
            if (visc) ((float *)e.f.dt_fac)[k] = (float)dtf_out;
            a2 = (double)fx * fx + (double)fy * fy + (double)fz * fz;
        } else {
            ((double *)e.f.au)[k] = acc[0];
            ((double *)e.f.av)[k] = acc[1];
            if (DIM == 3) ((double *)e.f.aw)[k] = acc[2];
            if (visc) ((double *)e.f.dt_fac)[k] = dtf_out;
            a2 = acc[0] * acc[0] + acc[1] * acc[1] + acc[2] * acc[2];
        }
        if (!isfinite(a2)) flag(e, SPHB_ST_NONFINITE_ACC);
    }
    if (!(mode & SPHB_FORCE_NO_MAXIMA)) {
        // one atomic per block and quantity (a block never spans two scenes)
        const double bdt = block_reduce(dtf_out, OpMax(), 0.0);
        const double ba2 = block_reduce(isfinite(a2) ? a2 : 0.0, OpMax(), 0.0);
        if (threadIdx.x == 0) {
            sphb_scene_state &sw = e.sstate[s];
            atomic_max_nonneg(&sw.max_dtfac, bdt);
            atomic_max_nonneg(&sw.max_acc2, ba2);
        }
    }
    // the integrator stage fused into the epilogue: the rates as stored
    // above, the new records (FP32C) or state (FP64) into the second copy.
    // In FP64 it replaces a launch of 3.5 us (5k particles) to 5.9 us (86k)
    // that re-reads the rates, for 1.5 to 2.3 us more of the pass: 5k drop 58.8
    // -> 55.7 us per step, 86k dam break 123 -> 116 us
    const int kind = ((mode & SPHB_FORCE_STAGE_MASK) >> 8) - 1;
    if (kind >= 0) {
        const bool stepped = (e.cfg.step_on >> a) & 1u;
        float d2 = 0.f;
        if (active && lane == 0 && (stepped || rm)) {
            const bool real = e.buf[cur].tag[k] == 0;
            auto stored = [](double v) { return F32 ? (double)(float)v : v; };
            double f[3], xv[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                f[d] = stored(acc[d]);
                xv[d] = stored(real ? xs[d] : 0.0);
            }
            const double dr = stored(real ? drho : 0.0);
            const float4 g_old =
                F32 ? ((const float4 *)e.f.geo)[k] : make_float4(0.f, 0.f, 0.f, 0.f);
            d2 = stage_particle<DIM, F32>(e, cur, k, s, a, kind, f, xm != 0u, xv, dr,
                                          F32 ? (float4 *)e.f.geo_next : nullptr,
                                          F32 ? e.f.vel_next : nullptr, g_old, !F32);
        }
        if (stepped && e.f.anchor) warp_max_disp(e, s, d2);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            // the particles move: the lists are not known to be complete
            // until the next rebin decision, and they leave the anchors
            e.work.meta[2] = 0;
            e.work.meta[3] = 0;
        }
    }
    block_add_u64(&e.work.pairs[1], np);
}

// CONT: the continuity scheme's pair terms too -- SPHDensityRate
// (density_funcs.pyx:119-156) and XSPHCorrection (xsph_funcs.pyx:40-86),
// each over its own sources, in the same traversal as the momentum.
// Register bounds, the list loops two entries ahead (four, or the records
// a batch ahead, lost at every bound; times of the pass with the density
// pass it overlaps): FP32C in 2D 72 (seven 128-thread blocks per SM; 332k
// dam break 3,778 us per 20 steps, 80 registers 3,966, 64 3,982; 256 drops
// 377 us a pass, 80 registers 418, 64 366), in 3D 80 (128^3 lattice's pressure
// gradient 597 us, 96 registers 671, 128 758), with the continuity terms 96
// (1,109 us per 10 steps of 146k particles, 80 registers 1,122, 128 1,163).
// FP64 in 2D 96: 16% of its 128-register time on an 86k-particle dam break
// was a second wave of blocks (1,304 -> 1,248 us per 10 steps).
// The FP64 pair is bound by the latency of its gathers and by issue: a batch's
// fields are loaded together, P / rho^2 is kept per particle, and no division
// or branch stands in a pair (one neighbour at a time with four dependent
// rounds of loads, eight divisions and a square root in branches: 134 us on
// that dam break, against 42).
template <int DIM, bool F32, bool CONT>
constexpr int force_regs()
{
    return F32 ? (CONT ? (DIM == 3 ? 128 : 96) : (DIM == 2 ? 72 : 80))
               : (DIM == 2 && !CONT ? 96 : 128);
}

template <int KT, int DIM, bool F32, int LANES, int R, bool CONT>
__global__ void __maxnreg__((force_regs<DIM, F32, CONT>()))
k_force(const __grid_constant__ sphb_engine e, int cur, uint32_t dest_mask,
        int with_gravity, int mode)
{
    // launched as a programmatic dependent of the density pass: everything
    // below reads what that pass wrote; the next rebin decision may launch
    // once every block of this pass has started
    pdl_wait();
    pdl_trigger();
    const sphb_tile tl = e.pair_tiles[blockIdx.x];
    const int A = e.cfg.num_arrays;
    const int s = tl.seg / A, a = tl.seg - s * A;
    const uint32_t mm = e.cfg.mom_src[a];
    const uint32_t rm = CONT ? e.cfg.rate_src[a] : 0u;
    const uint32_t xm = CONT ? e.cfg.xsph_src[a] : 0u;
    if (!((dest_mask >> a) & 1u) || (mm | rm | xm) == 0u) return;  // block-uniform
    // sources visited: those the lists hold (every pair function's); each
    // term keeps to its own sources when they differ
    const uint32_t src = CONT ? list_sources(e.cfg, a) : mm;
    const bool filt = CONT && ((mm && mm != src) || (rm && rm != src) || (xm && xm != src));
    const SegBounds seg(e, s);
    const int lane = threadIdx.x & (LANES - 1);
    const int k = tl.begin + (int)(threadIdx.x / LANES);
    const bool active = k < tl.end;
    const sphb_scene_state &st = e.sstate[s];
    const int n[3] = {st.n[0], st.n[1], st.n[2]};
    const int cell_base = st.cell_base, ncells = st.ncells;
    const sphb_scene &sc = e.scene[s];
    const int *__restrict__ start = e.work.start;
    const bool visc = (mode & 15) == 0;
    // split-form MonaghanArtificialViscosity alone (no pressure terms)
    const bool avisc = (mode & 15) == 2;
    // reuse the density pass's lists (recorded over list_sources); without
    // the per-source filter they must hold the momentum sources exactly
    const bool use_list = (mode & SPHB_FORCE_USE_LIST) && e.f.list_cap > 0 && e.f.nbr &&
                          e.f.nbr_cnt && (CONT || list_sources(e.cfg, a) == mm);
    unsigned int np = 0;   // pairs of this thread
    double acc[3] = {0.0, 0.0, 0.0};
    double dtf = 0.0;
    double drho = 0.0, xs[3] = {0.0, 0.0, 0.0};   // continuity scheme sums

    if constexpr (F32) {
        Kahan ax, ay, az;
        Kahan kr, kxx, kxy, kxz;   // density rate, XSPH velocity (CONT)
        float dtmax = 0.f, dt_h = 1.0f;   // dt_fac = dtmax dt_h
        if (active) {
            const int N = e.cfg.num_particles;
            const float4 *__restrict__ geo = (const float4 *)e.f.geo;
            const float *__restrict__ mass = (const float *)e.f.mass;
            const float4 *__restrict__ th = (const float4 *)e.f.thermo;
            const float csf = (float)sc.cell_size;
            const float4 gk = geo[k];
            const float4 tk = th[k];
            float uk, vk, wk = 0.f;
            if (DIM == 2) {
                const float2 vv = ((const float2 *)e.f.vel)[k];
                uk = vv.x;
                vk = vv.y;
            } else {
                const float4 vv = ((const float4 *)e.f.vel)[k];
                uk = vv.x;
                vk = vv.y;
                wk = vv.z;
            }
            const float xk = gk.x, yk = gk.y, zk = DIM == 3 ? gk.z : 0.f;
            const float hk = DIM == 3 ? gk.w : gk.z;
            const float rad = hk * (float)sc.radius_scale;
            const float rad2 = rad * rad;
            const float alpha = (float)sc.alpha, beta = (float)sc.beta;
            const float eta2 = (float)(sc.eta * sc.eta);
            const float kf = (float)Kern<KT>::template norm<DIM>();
            const float ihk = rcp_pair(hk);
            // fac / h of the dest: 2D kf/h^3, 3D kf/h^4
            const float fihk = DIM == 2 ? kf * ihk * ihk * ihk : kf * ihk * ihk * ihk * ihk;
            const float eh2k = mul_pair(eta2 * hk, hk);
            const float alp_k = alpha * hk, bet2_k = 2.0f * beta * hk * hk;
            // variable h: symmetric lists and, with hks, W and grad W
            // averaged over h_a and h_b (the AV and the CFL keep h_ab)
            const bool vh = sc.variable_h != 0, hks = sc.hks != 0;
            const float rsf = (float)sc.radius_scale;
            struct Rec {
                float4 g, t;
                float vx, vy, vz, m;
                uint32_t bit;   // the source's array as a mask bit (CONT)
            };
            auto load = [&](int j_) {
                Rec r;
                // list entries index the set (pads the dest itself); the
                // clamp only keeps a damaged list inside the arrays
                const int j = min(j_, N - 1);
                r.bit = filt ? 1u << seg.array_of(j) : ~0u;
                r.g = __ldg(geo + j);
                r.t = __ldg(th + j);
                r.m = DIM == 3 ? __ldg(mass + j) : r.g.w;
                if (visc || avisc || CONT) {
                    if (DIM == 2) {
                        const float2 vv = __ldg((const float2 *)e.f.vel + j);
                        r.vx = vv.x;
                        r.vy = vv.y;
                        r.vz = 0.f;
                    } else {
                        const float4 vv = __ldg((const float4 *)e.f.vel + j);
                        r.vx = vv.x;
                        r.vy = vv.y;
                        r.vz = vv.z;
                    }
                } else {
                    r.vx = r.vy = r.vz = 0.f;
                }
                return r;
            };
            auto pass = [&](auto uniform) {
                constexpr bool UH = decltype(uniform)::value;
                if (UH) dt_h = hk;
                // the pair body; with the force mode known at compile time
                // (KM = 0 MomentumEquation, 1 SPHPressureGradient, 2 the
                // split viscosity; -1 read at run time) the list loop
                // carries no test of it
                // The list loops (KM >= 0) evaluate every entry and have the
                // ones outside the support add 0 (list entries lie within the
                // support plus the skin, so few do): no branch separates the
                // entries of a batch.  The cell search branches.
                auto make_use = [&](auto known) {
                    constexpr int KM = decltype(known)::value;
                    const bool visc_k = KM < 0 ? visc : KM == 0;
                    const bool avisc_k = KM < 0 ? avisc : KM == 2;
                    return [&, visc_k, avisc_k](const Rec &r, float o, float dy, float dz) {
                        const float rx = fmaf(-o, csf, xk - r.g.x);
                        const float ry = fmaf(-dy, csf, yk - r.g.y);
                        float rz = 0.f;
                        float r2 = fmaf(ry, ry, mul_pair(rx, rx));
                        if (DIM == 3) {
                            rz = fmaf(-dz, csf, zk - r.g.z);
                            r2 = fmaf(rz, rz, r2);
                        }
                        const float hj = DIM == 3 ? r.g.w : r.g.z;
                        bool in = r2 < rad2;
                        if (!UH && vh) {
                            const float rj = hj * rsf;   // r < radius_scale max(h_a, h_b)
                            in = r2 < rad2 || r2 < rj * rj;
                        }
                        if (KM < 0 && !in) return;
                        np += in;
                        const bool mom_on = in && (!CONT || (mm & r.bit));
                        const bool rate_on = in && CONT && (rm & r.bit);
                        const bool xs_on = in && CONT && (xm & r.bit);
                        float hab = hk, eh2 = eh2k;
                        if (!UH) {
                            hab = 0.5f * (hk + hj);
                            eh2 = mul_pair(eta2 * hab, hab);
                        }
                        // P_a/rho_a^2 + P_b/rho_b^2 (none in the split viscosity)
                        float tmp = avisc_k ? 0.f : tk.w + r.t.w;
                        const float vx = uk - r.vx, vy = vk - r.vy, vz = wk - r.vz;
                        float dot = fmaf(vy, ry, mul_pair(vx, rx));
                        if (DIM == 3) dot = fmaf(vz, rz, dot);
                        // r = 0 (self) gives q = 0 and a finite gradient times r_ab = 0
                        const float ir = inv_dist(r2);
                        // grad W / r (and W for XSPH) at h_ab, or with hks the means
                        // of the values at h_a and h_b
                        float gw, w = 0.f;
                        if (UH) {
                            const float q = mul_pair(r2 * ir, ihk);
                            gw = Kern<KT>::template gw_in<false>(q, ir, ihk, fihk);
                            if (CONT) w = Kern<KT>::template w_in<false>(q, fihk * hk);
                        } else {
                            const float rr = r2 * ir;
                            auto at = [&](float hs, float &wh) {
                                const float ih = rcp_pair(hs);
                                const float fih = DIM == 2 ? kf * ih * ih * ih : kf * ih * ih * ih * ih;
                                const auto q = mul_pair(rr, ih);
                                if (CONT) wh = Kern<KT>::template w_in<true>(q, fih * hs);
                                return Kern<KT>::template gw_in<true>(q, ir, ih, fih);
                            };
                            float wa = 0.f, wb = 0.f;
                            if (hks) {
                                gw = 0.5f * (at(hk, wa) + at(hj, wb));
                                w = 0.5f * (wa + wb);
                            } else {
                                gw = at(hab, w);
                            }
                        }
                        if (CONT) {
                            // drho_a += m_b (v_a - v_b) . grad_a W
                            kr.add_prod(r.m, dot * gw, rate_on);
                            // XSPH: eps m_b W_ab (v_b - v_a) / rho_ab (eps at the end)
                            const float temp = r.m * w * rcp_pair(0.5f * (tk.x + r.t.x));
                            kxx.add_prod(-temp, vx, xs_on);
                            kxy.add_prod(-temp, vy, xs_on);
                            if (DIM == 3) kxz.add_prod(-temp, vz, xs_on);
                        }
                        if (visc_k || avisc_k) {
                            // mu / h_ab = dot / (r^2 + eta^2 h_ab^2); the factors
                            // h_ab go into alpha and beta
                            const float mu = dot * rcp_pair(r2 + eh2);
                            const float alp = UH ? alp_k : alpha * hab;
                            const float bet2 = UH ? bet2_k : 2.0f * beta * hab * hab;
                            // the split viscosity's dt_fac has 0.01 h_ab^2 written in
                            // (viscosity_funcs.pyx:103) whatever its eta
                            const float md =
                                avisc_k ? dot * rcp_pair(r2 + 0.01f * hab * hab) : mu;
                            dtmax = fmaxf(dtmax, mom_on ? fabsf(UH ? md : md * hab) : 0.f);
                            // Monaghan Pi_ab = (-alpha c_ab mu + beta mu^2) / rho_ab
                            // when v_ab . r_ab < 0, i.e. mu < 0; else 0: min(mu, 0)
                            // (the halves of c_ab and rho_ab cancel)
                            const float mn = fminf(mu, 0.f);
                            const float c2 = tk.z + r.t.z, rho2 = tk.x + r.t.x;
                            tmp = fmaf(mn * fmaf(bet2, mn, mul_pair(-alp, c2)), rcp_pair(rho2),
                                       tmp);
                        }
                        // (the products are selected, so a NaN outside the
                        // support stays there)
                        const float f = -r.m * tmp * gw;
                        ax.add_prod(f, rx, mom_on);
                        ay.add_prod(f, ry, mom_on);
                        if (DIM == 3) az.add_prod(f, rz, mom_on);
                    };
                };
                const int lc = list_count(e, use_list, k);
                if (lc >= 0) {
                    auto from_list = [&](auto known) {
                        auto use = make_use(known);
                        list_loop<LANES, 2>(
                            e, k, lane, lc, [&](uint32_t v) { return load(entry_index<DIM>(v)); },
                            [&](const Rec &r, uint32_t v) {
                                const EntryF en = entry_unpack_f<DIM>(v);
                                use(r, en.o, en.dy, en.dz);
                            });
                    };
                    switch (mode & 15) {   // block-uniform
                    case 0: from_list(std::integral_constant<int, 0>{}); break;
                    case 1: from_list(std::integral_constant<int, 1>{}); break;
                    default: from_list(std::integral_constant<int, 2>{}); break;
                    }
                    return;
                }
                auto use = make_use(std::integral_constant<int, -1>{});
                int cx, cy, cz;
                cell_coords(e.f.cell[k], n, cx, cy, cz);
                for_each_candidate<DIM, R, LANES>(
                    start, A, src, cell_base, ncells, n, cx, cy, cz, lane, N, e.work.status,
                    cell_trim_rel(e, xk, yk, zk, csf),
                    [&](int j, int o, int dy, int dz) {
                        use(load(j), (float)o, (float)dy, (float)dz);
                    });
            };
            if (sc.uniform_h) pass(std::true_type{});
            else pass(std::false_type{});
        }
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            ax.merge(__shfl_xor_sync(0xffffffffu, ax.sum, o), __shfl_xor_sync(0xffffffffu, ax.c, o));
            ay.merge(__shfl_xor_sync(0xffffffffu, ay.sum, o), __shfl_xor_sync(0xffffffffu, ay.c, o));
            if (DIM == 3)
                az.merge(__shfl_xor_sync(0xffffffffu, az.sum, o), __shfl_xor_sync(0xffffffffu, az.c, o));
            dtmax = fmaxf(dtmax, __shfl_xor_sync(0xffffffffu, dtmax, o));
        }
        acc[0] = ax.value();
        acc[1] = ay.value();
        acc[2] = az.value();
        dtf = dtmax * dt_h;
        if (CONT) {
#pragma unroll
            for (int o = LANES / 2; o > 0; o >>= 1) {
                kr.merge(__shfl_xor_sync(0xffffffffu, kr.sum, o), __shfl_xor_sync(0xffffffffu, kr.c, o));
                kxx.merge(__shfl_xor_sync(0xffffffffu, kxx.sum, o), __shfl_xor_sync(0xffffffffu, kxx.c, o));
                kxy.merge(__shfl_xor_sync(0xffffffffu, kxy.sum, o), __shfl_xor_sync(0xffffffffu, kxy.c, o));
                if (DIM == 3)
                    kxz.merge(__shfl_xor_sync(0xffffffffu, kxz.sum, o),
                              __shfl_xor_sync(0xffffffffu, kxz.c, o));
            }
            drho = kr.value();
            xs[0] = kxx.value() * sc.xsph_eps;
            xs[1] = kxy.value() * sc.xsph_eps;
            xs[2] = kxz.value() * sc.xsph_eps;
        }
    } else {
        double dt_h = 1.0;
        // fac / h of the gradients, applied to the sums where one serves all
        // pairs: a product and a constant fewer in the loop, whose 96 registers
        // spill (86k dam break 1,164 -> 1,146 us per 10 steps); w_scale: the
        // same for XSPH's W, with eps
        double scale = 1.0, w_scale = 1.0;
        if (active) {
            const int N = e.cfg.num_particles;
            const sphb_buffers &B = e.buf[cur];
            const double *__restrict__ rho = (const double *)e.f.rho;
            const double *__restrict__ pr = (const double *)e.f.p;
            const double *__restrict__ csnd = (const double *)e.f.cs;
            // P / rho^2 as the density pass and the Tait kernel left it; a
            // caller without the field has it taken per pair
            const double *__restrict__ prho2 = (const double *)e.f.thermo;
            const double xk = B.x[k], yk = B.y[k], zk = DIM == 3 ? B.z[k] : 0.0;
            const double uk = B.u[k], vk = B.v[k], wk = DIM == 3 ? B.w[k] : 0.0;
            const double hk = B.h[k];
            const double rhoa = rho[k], ca = csnd[k];
            auto p_rho2 = [&](int j) {
                if (prho2) return __ldg(prho2 + j);
                const double r = __ldg(rho + j);
                return __ldg(pr + j) * (1.0 / (r * r));
            };
            const double ta = p_rho2(k);
            const double rad = hk * sc.radius_scale;
            const double rad2 = __dmul_rn(rad, rad);
            const double alpha = sc.alpha, beta = sc.beta, eta2 = sc.eta * sc.eta;
            const double kf = Kern<KT>::template norm<DIM>();
            const double alp_k = alpha * hk, bet2_k = 2.0 * beta * hk * hk;
            const double ihk = rcp_pair(hk);
            const double fack = (DIM == 2 ? rcp_pair(hk * hk) : rcp_pair(hk * hk * hk)) * kf;
            const double fihk = fack * ihk;
            // with one h in the scene the symmetric set and the averaged
            // kernels are the plain ones
            const bool vh = sc.variable_h != 0, hks = sc.hks != 0;
            struct Rec {
                double x, y, z, u, v, w, m, h, rho, t, c;
                uint32_t bit;   // the source's array as a mask bit (CONT)
                bool ok;
            };
            auto pass = [&](auto uniform) {
                constexpr bool UH = decltype(uniform)::value;
                if (UH) dt_h = hk;
                if (UH) {
                    scale = fihk;
                    w_scale = fack * sc.xsph_eps;
                }
                // KM as in the FP32C body: the mode known at compile time in
                // the list loops, -1 in the cell search
                auto make_load = [&](auto known) {
                    constexpr int KM = decltype(known)::value;
                    return [&](int j, bool ok) {
                        Rec r;
                        r.ok = ok;
                        r.bit = filt ? 1u << seg.array_of(j) : ~0u;
                        r.x = __ldg(B.x + j);
                        r.y = __ldg(B.y + j);
                        r.z = DIM == 3 ? __ldg(B.z + j) : 0.0;
                        r.m = __ldg(B.m + j);
                        r.h = UH ? hk : __ldg(B.h + j);
                        r.t = KM == 2 ? 0.0 : p_rho2(j);
                        r.u = r.v = r.w = r.rho = r.c = 0.0;
                        if (KM != 1 || CONT) {
                            r.u = __ldg(B.u + j);
                            r.v = __ldg(B.v + j);
                            if (DIM == 3) r.w = __ldg(B.w + j);
                            r.rho = __ldg(rho + j);
                        }
                        if (KM != 1) r.c = __ldg(csnd + j);
                        return r;
                    };
                };
                auto make_use = [&](auto known) {
                    constexpr int KM = decltype(known)::value;
                    const bool visc_k = KM < 0 ? visc : KM == 0;
                    const bool avisc_k = KM < 0 ? avisc : KM == 2;
                    return [&, visc_k, avisc_k](const Rec &r) {
                        const double rx = xk - r.x, ry = yk - r.y;
                        const double rz = DIM == 3 ? zk - r.z : 0.0;
                        const double r2 = dist2_ref<DIM>(rx, ry, rz);
                        double radj2 = rad2;
                        if (!UH && vh) {
                            // symmetric: r^2 < (radius_scale h_a)^2 or (radius_scale h_b)^2
                            const double rj = r.h * sc.radius_scale;
                            radj2 = fmax(rad2, __dmul_rn(rj, rj));
                        }
                        const bool in = r.ok && r2 < radj2;
                        if (KM < 0 && !in) return;
                        np += in;
                        const bool mom_on = in && (!CONT || (mm & r.bit));
                        const bool rate_on = in && CONT && (rm & r.bit);
                        const bool xs_on = in && CONT && (xm & r.bit);
                        const double hab = UH ? hk : 0.5 * (hk + r.h);
                        double ir;
                        const double rr = dist_pair(r2, ir);
                        // the quotient's residual matters to W, whose sum XSPH is,
                        // not to the gradients' (accelerations 0.71 of the error
                        // of divisions and square roots with it and without)
                        auto q_of = [](double r, double h, double ih) {
                            return CONT ? over_h(r, h, ih) : mul_pair(r, ih);
                        };
                        // grad W / r (and W for XSPH) at h_ab, or with hks the
                        // means of the values at h_a and h_b (pressure_funcs.pyx:
                        // 371-381)
                        double gw, w = 0.0;
                        if (UH) {
                            const double q = q_of(rr, hk, ihk);
                            gw = Kern<KT>::template gw_in<false>(q, ir, ihk, 1.0);
                            if (CONT) w = Kern<KT>::template w_in<false>(q, 1.0);
                        } else {
                            auto eval = [&](double hs, double ih, double fac, double fih,
                                            double &wh) {
                                const double q = q_of(rr, hs, ih);
                                if (CONT) wh = Kern<KT>::template w_in<true>(q, fac);
                                return Kern<KT>::template gw_in<true>(q, ir, ih, fih);
                            };
                            auto at = [&](double hs, double &wh) {
                                const double ih = rcp_pair(hs);
                                const double fac =
                                    (DIM == 2 ? rcp_pair(hs * hs) : rcp_pair(hs * hs * hs)) * kf;
                                return eval(hs, ih, fac, fac * ih, wh);
                            };
                            double wa = 0.0, wb = 0.0;
                            if (hks) {
                                gw = 0.5 * (eval(hk, ihk, fack, fihk, wa) + at(r.h, wb));
                                w = 0.5 * (wa + wb);
                            } else {
                                gw = at(hab, w);
                            }
                        }
                        const double gx = rx * gw, gy = ry * gw, gz = rz * gw;
                        const double vx = uk - r.u, vy = vk - r.v, vz = wk - r.w;
                        if (CONT) {
                            // SPHDensityRate: ((v_a - v_b) . grad_a W) m_b
                            double d = vx * gx + vy * gy;
                            if (DIM == 3) d += vz * gz;
                            drho += rate_on ? d * r.m : 0.0;
                            // XSPHCorrection: m_b W_ab / rho_ab (v_b - v_a) eps
                            // (eps with the normalisation, at the end, where one
                            // serves all pairs)
                            double temp = r.m * w * rcp_pair(0.5 * (r.rho + rhoa));
                            if (!UH) temp *= sc.xsph_eps;
                            xs[0] -= xs_on ? temp * vx : 0.0;
                            xs[1] -= xs_on ? temp * vy : 0.0;
                            if (DIM == 3) xs[2] -= xs_on ? temp * vz : 0.0;
                        }
                        // P_a/rho_a^2 + P_b/rho_b^2; the split viscosity has none
                        // (tmp = piab; tmp *= -mb, viscosity_funcs.pyx:125-126)
                        double tmp = avisc_k ? 0.0 : ta + r.t;
                        if (visc_k || avisc_k) {
                            double dot = vx * rx + vy * ry;
                            if (DIM == 3) dot += vz * rz;
                            const double mu = dot * rcp_pair(r2 + eta2 * hab * hab);
                            const double alp = UH ? alp_k : alpha * hab;
                            const double bet2 = UH ? bet2_k : 2.0 * beta * hab * hab;
                            const double md =
                                avisc_k ? dot * rcp_pair(r2 + 0.01 * hab * hab) : mu;
                            dtf = fmax(dtf, mom_on ? fabs(UH ? md : md * hab) : 0.0);
                            // Monaghan Pi_ab when v_ab . r_ab < 0, selected, not branched on
                            const double c2 = ca + r.c, rho2 = rhoa + r.rho;
                            const double piab = mu * fma(bet2, mu, -alp * c2) * rcp_pair(rho2);
                            tmp += dot < 0.0 ? piab : 0.0;
                        }
                        tmp *= -r.m;
                        acc[0] += mom_on ? tmp * gx : 0.0;
                        acc[1] += mom_on ? tmp * gy : 0.0;
                        if (DIM == 3) acc[2] += mom_on ? tmp * gz : 0.0;
                    };
                };
                const int lc = list_count(e, use_list, k);
                if (lc >= 0) {
                    auto from_list = [&](auto known) {
                        auto load = make_load(known);
                        auto use = make_use(known);
                        list_loop<LANES, 2>(
                            e, k, lane, lc,
                            [&](uint32_t v) {
                                int j;
                                const bool ok = list_entry_d<DIM>(e, v, k, j);
                                return load(j, ok);
                            },
                            [&](const Rec &r, uint32_t) { use(r); });
                    };
                    switch (mode & 15) {   // block-uniform
                    case 0: from_list(std::integral_constant<int, 0>{}); break;
                    case 1: from_list(std::integral_constant<int, 1>{}); break;
                    default: from_list(std::integral_constant<int, 2>{}); break;
                    }
                    return;
                }
                auto load = make_load(std::integral_constant<int, -1>{});
                auto use = make_use(std::integral_constant<int, -1>{});
                int cx, cy, cz;
                cell_coords(e.f.cell[k], n, cx, cy, cz);
                for_each_candidate<DIM, R, LANES>(
                    start, A, src, cell_base, ncells, n, cx, cy, cz, lane, N, e.work.status,
                    cell_trim_abs<DIM>(e, st, sc.cell_size, xk, yk, zk, cx, cy, cz),
                    [&](int j, int, int, int) { use(load(j, true)); });
            };
            if (sc.uniform_h) pass(std::true_type{});
            else pass(std::false_type{});
        }
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
            acc[1] += __shfl_xor_sync(0xffffffffu, acc[1], o);
            if (DIM == 3) acc[2] += __shfl_xor_sync(0xffffffffu, acc[2], o);
            dtf = fmax(dtf, __shfl_xor_sync(0xffffffffu, dtf, o));
            if (CONT) {
                drho += __shfl_xor_sync(0xffffffffu, drho, o);
                for (int d = 0; d < DIM; ++d) xs[d] += __shfl_xor_sync(0xffffffffu, xs[d], o);
            }
        }
        dtf *= dt_h;
#pragma unroll
        for (int d = 0; d < DIM; ++d) acc[d] *= scale;
        if (CONT) {
            drho *= scale;
#pragma unroll
            for (int d = 0; d < DIM; ++d) xs[d] *= w_scale;
        }
    }

    force_finish<DIM, F32, CONT>(e, cur, k, s, a, active, lane, acc, dtf, drho, xs,
                                 visc || avisc, mm, rm, xm, with_gravity, mode, np);
}

template <int KT, int DIM, bool F32, int LV, int RV>
static void launch_force_lr(const sphb_engine &e, int cur, uint32_t dm, int grav, int mode,
                            bool cont, cudaStream_t st)
{
    const dim3 g(e.num_pair_tiles), b(e.cfg.pair_block);
    if (cont) launch_pdl(k_force<KT, DIM, F32, LV, RV, true>, g, b, 0, st, e, cur, dm, grav, mode);
    else launch_pdl(k_force<KT, DIM, F32, LV, RV, false>, g, b, 0, st, e, cur, dm, grav, mode);
}

template <int KT, int DIM, bool F32>
static void launch_force_p(const sphb_engine &e, int cur, uint32_t dm, int grav,
                           int mode, cudaStream_t st)
{
    bool cont = false;
    for (int a = 0; a < SPHB_MAX_ARRAYS; ++a) cont = cont || e.cfg.rate_src[a] || e.cfg.xsph_src[a];
#define SPHB_L(LV, RV) launch_force_lr<KT, DIM, F32, LV, RV>(e, cur, dm, grav, mode, cont, st)
    switch (e.cfg.lanes * 10 + e.cfg.stencil) {
    case 11: SPHB_L(1, 1); break;
    case 12: SPHB_L(1, 2); break;
    case 21: SPHB_L(2, 1); break;
    case 22: SPHB_L(2, 2); break;
    case 41: SPHB_L(4, 1); break;
    case 42: SPHB_L(4, 2); break;
    case 81: SPHB_L(8, 1); break;
    case 82: SPHB_L(8, 2); break;
    }
#undef SPHB_L
}

template <int KT, int DIM>
void launch_force_kt(const sphb_engine &e, int cur, uint32_t dm, int grav, int mode,
                     cudaStream_t st)
{
    if constexpr (DIM == 2) {
        if (e.cfg.pair_mode == SPHB_PAIRS_TILED) {
            launch_force_tiled<KT>(e, cur, dm, grav, mode, st);
            return;
        }
    }
    if (e.cfg.precision == SPHB_FP32C) launch_force_p<KT, DIM, true>(e, cur, dm, grav, mode, st);
    else launch_force_p<KT, DIM, false>(e, cur, dm, grav, mode, st);
}

}  // namespace sphb
