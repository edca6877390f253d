// sphb_density_pass.cuh -- the summation-density pass (SPHRho + Tait
// epilogue, neighbour-list recording), templated on the smoothing kernel.
// Included by one translation unit per kernel type (sphb_pass_*.cu), which
// instantiates launch_density_kt for its kernel and dimensions.
//
// SPHRho (S/sph/funcs/density_funcs.pyx:37-73; OpenCL S/sph/funcs/
// density_funcs.clt:3-53): rho_a = sum_b m_b W(r_ab, (h_a + h_b)/2) over the
// neighbours r_ab^2 < (radius_scale h_a)^2 of every source array, self
// included.  TaitEquation (S/sph/funcs/eos_funcs.pyx:88-129): p =
// B((rho/rho0)^gamma-1), cs = c0 (rho/rho0)^((gamma-1)/2), fused as the
// epilogue.  Non-LocalReal dests get 0 (S/sph/sph_func.pyx:220-227).
//
// FP32C: pair geometry in FP32 from cell-relative positions, the sum in FP32
// with Kahan compensation, the EOS in FP64.  FP64: the reference's neighbour
// predicate, operation for operation; its kernels with the reciprocals of
// sphb_kernels.cuh in place of divisions and square roots.  Against 80-bit
// arithmetic the density of a drop of 60k particles with varying h is 1.2e-16
// off; summed one pair after the other with divisions and square roots it
// was 1.45e-16 off.
//
// Variable smoothing length (scene.variable_h): the neighbours are the
// symmetric set of VarHNbrParticleLocator (S/base/nnps.pyx:691-786),
// r^2 < (radius_scale h_a)^2 or r^2 < (radius_scale h_b)^2.  With scene.hks
// the pair's W is the mean of W(r, h_a) and W(r, h_b) (density_funcs.pyx:
// 56-63) instead of W(r, (h_a + h_b) / 2).

#pragma once

#include <type_traits>

#include "sphb_kernels.cuh"
#include "sphb_launch.cuh"
#include "sphb_pairs.cuh"

namespace sphb {

// The outputs of dest k after its density sum: rho (0 for non-LocalReal
// dests), the Tait EOS when asked and the array is a Tait dest, the FP32C
// record {rho, p, cs, p / rho^2}, and the pair count.  Every thread of the
// block calls it; rho is valid in lane 0 of each dest.
template <bool F32>
__device__ __forceinline__ void density_finish(const sphb_engine &e, int cur, int k, int s, int a,
                                               bool active, int lane, double rho, int with_eos,
                                               unsigned int np)
{
    const sphb_scene &sc = e.scene[s];
    if (active && lane == 0) {
        const bool real = e.buf[cur].tag[k] == 0;
        if (!real) rho = 0.0;
        const bool eos = with_eos && ((e.cfg.tait_on >> a) & 1u);
        double p = 0.0, c = 0.0;
        if (eos && real) {
            const double ratio = rho / sc.rho0;
            p = (eos_pow<F32>(ratio, sc.gamma) - 1.0) * sc.B;
            c = eos_pow<F32>(ratio, 0.5 * (sc.gamma - 1.0)) * sc.c0;
        }
        if constexpr (F32) {
            float4 *th = (float4 *)e.f.thermo;
            float4 t = th[k];
            t.x = (float)rho;
            if (eos) {
                t.y = (float)p;
                t.z = (float)c;
            }
            t.w = t.x != 0.f ? t.y / (t.x * t.x) : 0.f;
            th[k] = t;
            if (!isfinite(t.x) || !isfinite(t.y)) flag(e, SPHB_ST_NONFINITE_RHO);
        } else {
            ((double *)e.f.rho)[k] = rho;
            if (eos) {
                ((double *)e.f.p)[k] = p;
                ((double *)e.f.cs)[k] = c;
            }
            // the force pass's P / rho^2, once per particle instead of per pair
            if (e.f.thermo && e.f.p)
                ((double *)e.f.thermo)[k] = (eos ? p : ((double *)e.f.p)[k]) * (1.0 / (rho * rho));
            if (!isfinite(rho) || !isfinite(p)) flag(e, SPHB_ST_NONFINITE_RHO);
        }
    }
    block_add_u64(&e.work.pairs[0], np);
}

// The 2D FP32C variants are held to 48 registers, five 256-thread blocks per
// SM (62 registers and four blocks otherwise): 2-12% shorter passes on the
// dam break, the list-recording pass gaining most.  The 3D FP32C variants are
// held to four blocks (64 registers) and the FP64 ones to three (80; they
// would take 86 and fit two).
template <int KT, int DIM, bool F32, int LANES, int R>
__global__ void __launch_bounds__(256, F32 ? (DIM == 2 ? 5 : 4) : 3)
k_density(const __grid_constant__ sphb_engine e, int cur, uint32_t dest_mask, int flags)
{
    // launched as a programmatic dependent of the rebin before it: the cells,
    // records and lists are read only after this; the force pass that
    // follows may launch once every block has started
    pdl_wait();
    pdl_trigger();
    const int with_eos = flags & SPHB_DENSITY_EOS;
    // list reuse: read the lists when the last rebin decision kept them
    // (work.meta[2]); otherwise record them, with the skin
    const bool reuse = (flags & SPHB_DENSITY_LIST_IF_VALID) && e.f.list_cap > 0;
    const bool from_list = e.f.list_cap > 0 && ((flags & SPHB_DENSITY_USE_LIST) ||
                                                (reuse && e.work.meta[2] == 1));
    // lists only (continuity scheme): record the lists after a rebin, no
    // density; with the lists kept there is nothing to do
    const bool lists_only = (flags & SPHB_DENSITY_LISTS_ONLY) != 0;
    const sphb_tile tl = e.pair_tiles[blockIdx.x];
    const int A = e.cfg.num_arrays;
    const int s = tl.seg / A, a = tl.seg - s * A;
    const uint32_t rsrc = e.cfg.rho_src[a];           // SPHRho sources
    const uint32_t lsrc = list_sources(e.cfg, a);     // sources the lists hold
    if (!((dest_mask >> a) & 1u) || (lists_only ? lsrc : rsrc) == 0u) return;  // block-uniform
    if (lists_only && (from_list || e.f.list_cap == 0)) return;
    // recording, or reading the lists: every list source; a cell search
    // without recording: the SPHRho sources alone
    const bool records = e.f.list_cap > 0 && !from_list;
    const uint32_t src = (records || from_list) ? lsrc : rsrc;
    // neighbours outside the SPHRho sources are skipped by the sum
    const bool filt = src != rsrc;
    const SegBounds seg(e, s);
    const int lane = threadIdx.x & (LANES - 1);
    const int k = tl.begin + (int)(threadIdx.x / LANES);
    const bool active = k < tl.end;
    const sphb_scene_state &st = e.sstate[s];
    const int n[3] = {st.n[0], st.n[1], st.n[2]};
    const int cell_base = st.cell_base, ncells = st.ncells;
    const sphb_scene &sc = e.scene[s];
    const int *__restrict__ start = e.work.start;
    unsigned int np = 0;   // pairs of this thread
    double rho = 0.0;
    // neighbour list of this dest, recorded (unless this pass reads them)
    // with the skin when it is meant for reuse
    const int N = e.cfg.num_particles;
    uint32_t *nbr = (e.f.list_cap > 0 && !from_list) ? e.f.nbr : nullptr;
    const double skin = (nbr && reuse) ? sc.skin_max : 0.0;
    if (nbr && blockIdx.x == 0 && threadIdx.x == 0) {
        // reusable only when recorded with the skin at the anchors (the
        // positions of the last rebin, work.meta[3] == 2); no pass of this
        // kernel reads meta[4], and a plain record also withdraws meta[2]
        e.work.meta[4] = (reuse && e.work.meta[3] == 2) ? 1 : 0;
        if (!reuse) e.work.meta[2] = 0;
    }
    int recorded = -1;   // entries of the list (-1: overflow, or none recorded)

    extern __shared__ int2 s_rows[];   // record_list's row ranges
    // FP32C in 2D with cells of the whole reach: summing while searching
    // saves the second look at the lists (442 against 474 us, the recording
    // pass of 256 drops); with cells of half the reach, in 3D, in FP64 and
    // for the wide quintic the sum over the recorded list is shorter (3D
    // cube of 64k 145 -> 93 us, FP64 dam break of 86k 38.6 -> 34.1 us,
    // quintic drop of 50k 55.6 -> 50.0 us)
    constexpr bool ONE_PHASE =
        F32 && DIM == 2 && R == 1 && LANES == 1 && KT != SPHB_KERNEL_QUINTIC;
    const int kq = active ? k : tl.begin;   // inactive threads read a valid particle
    if constexpr (F32) {
        Kahan acc;
        const float4 *__restrict__ geo = (const float4 *)e.f.geo;
        const float *__restrict__ mass = (const float *)e.f.mass;
        const float4 gk = geo[kq];
        const float csf = (float)sc.cell_size;
        const float xk = gk.x, yk = gk.y, zk = DIM == 3 ? gk.z : 0.f;
        const float hk = DIM == 3 ? gk.w : gk.z;
        const float rad = hk * (float)sc.radius_scale;
        const float rad2 = rad * rad;
        // variable h: symmetric lists and, with hks, W averaged over h_a, h_b
        const bool vh = sc.variable_h != 0, hks = sc.hks != 0;
        const float rsf = (float)sc.radius_scale;
        // a candidate of the list: within the support (the larger of the two
        // with variable h) plus the skin
        const float radl = (float)((hk * sc.radius_scale + skin) * (1.0 + 1e-5));
        const float radl2 = radl * radl;
        const float skinf = (float)skin;
        auto listed = [&](float r2, float hj, bool sym) {
            const float rl = (hj * rsf + skinf) * (1.0f + 1e-5f);
            return r2 < (sym ? fmaxf(radl2, rl * rl) : radl2);
        };
        auto dist2_to = [&](const float4 &g, float o, float dy, float dz) {
            const float dx = fmaf(-o, csf, xk - g.x);
            const float ddy = fmaf(-dy, csf, yk - g.y);
            float r2 = fmaf(ddy, ddy, mul_pair(dx, dx));
            if (DIM == 3) {
                const float ddz = fmaf(-dz, csf, zk - g.z);
                r2 = fmaf(ddz, ddz, r2);
            }
            return r2;
        };
        if constexpr (LANES > 1) {
            if (nbr) {
                const int local = e.f.cell[kq];
                int cx, cy, cz;
                cell_coords(local, n, cx, cy, cz);
                recorded = record_list<DIM, R, LANES>(
                    e, nbr, s_rows, k, active, src, cell_base, ncells, n, local, cx, cy, cz,
                    cell_trim_rel(e, xk, yk, zk, csf), [&](int j, int o, int dy, int dz) {
                        const float4 g = __ldg(geo + j);
                        return listed(dist2_to(g, (float)o, (float)dy, (float)dz),
                                      DIM == 3 ? g.w : g.z, vh);
                    });
            }
        }
        if (active) {
            const float kf = (float)Kern<KT>::template norm<DIM>();
            const float ihk = rcp_pair(hk);
            const float fack = DIM == 2 ? kf * ihk * ihk : kf * ihk * ihk * ihk;
            struct Rec {
                float4 g;
                float m;
                bool ok;
            };
            // list entries index the set (pads the dest itself); the clamp
            // only keeps a damaged list inside the arrays
            auto load = [&](int j_) {
                Rec r;
                const int j = min(j_, N - 1);
                r.ok = !filt || ((rsrc >> seg.array_of(j)) & 1u);
                r.g = __ldg(geo + j);
                r.m = DIM == 3 ? __ldg(mass + j) : r.g.w;
                return r;
            };
            // uniform h (every particle of the scene): h_ab = h_a, and the
            // kernel's 1/h and normalisation are the dest's
            auto pass = [&](auto uniform) {
                constexpr bool UH = decltype(uniform)::value;
                // flat: the list loops' form, every entry evaluated and the
                // ones outside the support adding 0 (list entries lie within
                // the support plus the skin, so few do), which leaves no
                // branch between the entries of a batch
                auto use = [&](const Rec &r, float r2, auto flat) {
                    const float hj = DIM == 3 ? r.g.w : r.g.z;
                    bool in = !lists_only && r.ok && r2 < rad2;
                    if (!UH && vh) {
                        const float rj = hj * rsf;   // r < radius_scale max(h_a, h_b)
                        in = !lists_only && r.ok && (r2 < rad2 || r2 < rj * rj);
                    }
                    if (!decltype(flat)::value && !in) return;
                    const float ir = inv_dist(r2);   // q = 0 at r = 0
                    float w;
                    if (UH) {
                        w = Kern<KT>::template w_in<false>(mul_pair(r2 * ir, ihk), fack);
                    } else {
                        // W(r, h_ab), or with hks (W(r, h_a) + W(r, h_b)) / 2
                        const float rr = r2 * ir;
                        auto w_at = [&](float hs) {
                            const float ih = rcp_pair(hs);
                            return Kern<KT>::template w_in<true>(
                                mul_pair(rr, ih), DIM == 2 ? kf * ih * ih : kf * ih * ih * ih);
                        };
                        w = hks ? 0.5f * (w_at(hk) + w_at(hj)) : w_at(0.5f * (hk + hj));
                    }
                    acc.add_prod(r.m, w, in);
                    np += in;
                };
                // the common case (one h, every source summed, densities
                // wanted) with the tests that cannot fail there out of the
                // loops: the same arithmetic as load() and use()
                const bool plain = UH && !filt && !lists_only;
                auto load_all = [&](int j_) {
                    Rec r;
                    const int j = min(j_, N - 1);
                    r.ok = true;
                    r.g = __ldg(geo + j);
                    r.m = DIM == 3 ? __ldg(mass + j) : r.g.w;
                    return r;
                };
                auto sum_plain = [&](const Rec &r, float r2) {
                    const bool in = r2 < rad2;
                    const float ir = inv_dist(r2);   // q = 0 at r = 0
                    const float w = Kern<KT>::template w_in<false>(mul_pair(r2 * ir, ihk), fack);
                    acc.add_prod(r.m, w, in);
                    np += in;
                };
                if constexpr (LANES == 1) {
                    if (nbr) {
                        // one thread a dest: record, then sum over the list
                        // just written, whose entries are nearly all
                        // neighbours (candidates are 15 to 50% of the time);
                        // ONE_PHASE sums while it searches
                        ListWriter<DIM, 1> list(nbr, k, e);
                        int cx, cy, cz;
                        cell_coords(e.f.cell[k], n, cx, cy, cz);
                        for_each_candidate<DIM, R, 1>(
                            start, A, src, cell_base, ncells, n, cx, cy, cz, lane, N,
                            e.work.status, cell_trim_rel(e, xk, yk, zk, csf),
                            [&](int j, int o, int dy, int dz) {
                                const float4 g = __ldg(geo + j);
                                float r2;
                                if (ONE_PHASE) {
                                    r2 = dist2_to(g, (float)o, (float)dy, (float)dz);
                                } else {
                                    // (not summed: contracted as the compiler
                                    // likes, 1,498 -> 1,416 us on a 128^3 lattice)
                                    const float dx = (xk - g.x) - (float)o * csf;
                                    const float ddy = (yk - g.y) - (float)dy * csf;
                                    r2 = dx * dx + ddy * ddy;
                                    if (DIM == 3) {
                                        const float ddz = (zk - g.z) - (float)dz * csf;
                                        r2 += ddz * ddz;
                                    }
                                }
                                list.put(listed(r2, DIM == 3 ? g.w : g.z, !UH && vh), j, o, dy,
                                         dz);
                                if (ONE_PHASE) {
                                    const Rec r{g, g.w, !filt || ((rsrc >> seg.array_of(j)) & 1u)};
                                    use(r, r2, std::false_type{});
                                }
                            });
                        recorded = list.finish(k);
                        if (ONE_PHASE || lists_only) return;
                    }
                }
                if (lists_only) return;
                // the list just recorded, or the kept one
                const int cnt = nbr ? recorded : list_count(e, from_list, k);
                if (cnt >= 0) {
                    auto dist2 = [&](const Rec &r, uint32_t v) {
                        const EntryF en = entry_unpack_f<DIM>(v);
                        return dist2_to(r.g, en.o, en.dy, en.dz);
                    };
                    if (plain)
                        list_loop<LANES, 4>(
                            e, k, lane, cnt,
                            [&](uint32_t v) { return load_all(entry_index<DIM>(v)); },
                            [&](const Rec &r, uint32_t v) {
                                sum_plain(r, dist2(r, v));
                            });
                    else
                        list_loop<LANES, 4>(
                            e, k, lane, cnt,
                            [&](uint32_t v) { return load(entry_index<DIM>(v)); },
                            [&](const Rec &r, uint32_t v) {
                                use(r, dist2(r, v), std::true_type{});
                            });
                    return;
                }
                int cx, cy, cz;
                cell_coords(e.f.cell[k], n, cx, cy, cz);
                for_each_candidate<DIM, R, LANES>(
                    start, A, src, cell_base, ncells, n, cx, cy, cz, lane, N, e.work.status,
                    cell_trim_rel(e, xk, yk, zk, csf), [&](int j, int o, int dy, int dz) {
                        const Rec r = load(j);
                        use(r, dist2_to(r.g, (float)o, (float)dy, (float)dz),
                            std::false_type{});
                    });
            };
            if (sc.uniform_h) pass(std::true_type{});
            else pass(std::false_type{});
        }
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            const float os = __shfl_xor_sync(0xffffffffu, acc.sum, o);
            const float oc = __shfl_xor_sync(0xffffffffu, acc.c, o);
            acc.merge(os, oc);
        }
        rho = acc.value();
    } else {
        // two sums, taken in turn: half the roundings in each (that density:
        // 1.5e-16 off with one) at no more operations
        double sum = 0.0, next = 0.0;
        const sphb_buffers &B = e.buf[cur];
        const double xk = B.x[kq], yk = B.y[kq], zk = DIM == 3 ? B.z[kq] : 0.0;
        const double hk = B.h[kq];
        const double rad = hk * sc.radius_scale;
        const double rad2 = __dmul_rn(rad, rad);
        // with one h in the scene the symmetric set and the averaged kernel
        // are the plain ones
        const bool vh = sc.variable_h != 0, hks = sc.hks != 0;
        const double radl = (rad + skin) * (1.0 + 1e-5);
        const double radl2 = radl * radl;
        auto accept = [&](int j, auto sym) {
            const double d2 = dist2_ref<DIM>(xk - __ldg(B.x + j), yk - __ldg(B.y + j),
                                             DIM == 3 ? zk - __ldg(B.z + j) : 0.0);
            if (!decltype(sym)::value) return d2 < radl2;
            const double rl = (__ldg(B.h + j) * sc.radius_scale + skin) * (1.0 + 1e-5);
            return d2 < fmax(radl2, rl * rl);
        };
        auto record = [&](auto sym) {
            const int local = e.f.cell[kq];
            int cx, cy, cz;
            cell_coords(local, n, cx, cy, cz);
            const CellTrim trim = cell_trim_abs<DIM>(e, st, sc.cell_size, xk, yk, zk, cx, cy, cz);
            if constexpr (LANES > 1) {
                recorded = record_list<DIM, R, LANES>(
                    e, nbr, s_rows, k, active, src, cell_base, ncells, n, local, cx, cy, cz, trim,
                    [&](int j, int, int, int) { return accept(j, sym); });
            } else if (active) {
                ListWriter<DIM, 1> list(nbr, k, e);
                for_each_candidate<DIM, R, 1>(
                    start, A, src, cell_base, ncells, n, cx, cy, cz, lane, N, e.work.status, trim,
                    [&](int j, int o, int oy, int oz) {
                        list.put(accept(j, sym), j, o, oy, oz);
                    });
                recorded = list.finish(k);
            }
        };
        if (nbr) {   // block-uniform, as is what the scene says of h
            if (vh && !sc.uniform_h) record(std::true_type{});
            else record(std::false_type{});
        }
        if (active && !(lists_only && nbr)) {
            const double kf = Kern<KT>::template norm<DIM>();
            const double ihk = rcp_pair(hk);
            const double fack = (DIM == 2 ? rcp_pair(hk * hk) : rcp_pair(hk * hk * hk)) * kf;
            struct Rec {
                double x, y, z, m, h;
                bool ok;
            };
            auto pass = [&](auto uniform) {
                constexpr bool UH = decltype(uniform)::value;
                auto load = [&](int j, bool ok) {
                    Rec r;
                    r.ok = ok && (!filt || ((rsrc >> seg.array_of(j)) & 1u));
                    r.x = __ldg(B.x + j);
                    r.y = __ldg(B.y + j);
                    r.z = DIM == 3 ? __ldg(B.z + j) : 0.0;
                    r.m = __ldg(B.m + j);
                    r.h = UH ? hk : __ldg(B.h + j);
                    return r;
                };
                auto dist2 = [&](const Rec &r) {
                    return dist2_ref<DIM>(xk - r.x, yk - r.y, DIM == 3 ? zk - r.z : 0.0);
                };
                auto use = [&](const Rec &r, double d2, auto flat) {
                    // symmetric: r^2 < (radius_scale h_a)^2 or (radius_scale h_b)^2
                    double radj2 = rad2;
                    if (!UH && vh) {
                        const double rj = r.h * sc.radius_scale;
                        radj2 = fmax(rad2, __dmul_rn(rj, rj));
                    }
                    const bool in = r.ok && d2 < radj2;
                    if (!decltype(flat)::value && !in) return;
                    double ir, w;
                    const double rr = dist_pair(d2, ir);
                    if (UH) {
                        w = Kern<KT>::template w_in<false>(over_h(rr, hk, ihk), fack);
                    } else {
                        // W(r, h_ab), or with hks (W(r, h_a) + W(r, h_b)) / 2
                        auto w_at = [&](double hs) {
                            const double ih = rcp_pair(hs);
                            return Kern<KT>::template w_in<true>(
                                over_h(rr, hs, ih),
                                (DIM == 2 ? rcp_pair(hs * hs) : rcp_pair(hs * hs * hs)) * kf);
                        };
                        w = hks ? 0.5 * (Kern<KT>::template w_in<true>(over_h(rr, hk, ihk), fack) +
                                         w_at(r.h))
                                : w_at(0.5 * (hk + r.h));
                    }
                    const double add = sum + (in ? r.m * w : 0.0);
                    sum = next;
                    next = add;
                    np += in;
                };
                const int cnt = nbr ? recorded : list_count(e, from_list, k);
                if (cnt >= 0) {
                    list_loop<LANES, 4>(
                        e, k, lane, cnt,
                        [&](uint32_t v) {
                            int j;
                            const bool ok = list_entry_d<DIM>(e, v, k, j);
                            return load(j, ok);
                        },
                        [&](const Rec &r, uint32_t) { use(r, dist2(r), std::true_type{}); });
                    return;
                }
                int cx, cy, cz;
                cell_coords(e.f.cell[k], n, cx, cy, cz);
                for_each_candidate<DIM, R, LANES>(
                    start, A, src, cell_base, ncells, n, cx, cy, cz, lane, N, e.work.status,
                    cell_trim_abs<DIM>(e, st, sc.cell_size, xk, yk, zk, cx, cy, cz),
                    [&](int j, int, int, int) {
                        const Rec r = load(j, true);
                        use(r, dist2(r), std::false_type{});
                    });
            };
            if (sc.uniform_h) pass(std::true_type{});
            else pass(std::false_type{});
        }
        sum += next;
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        rho = sum;
    }

    if (active && nbr && lane == 0) e.f.nbr_cnt[k] = recorded;
    density_finish<F32>(e, cur, k, s, a, active && !lists_only, lane, rho, with_eos, np);
}

template <int KT, int DIM, bool F32>
static void launch_density_p(const sphb_engine &e, int cur, uint32_t dm, int eos,
                             cudaStream_t st)
{
    const dim3 g(e.num_pair_tiles), b(e.cfg.pair_block);
#define SPHB_L(LV, RV)                                                                   \
    launch_pdl(k_density<KT, DIM, F32, LV, RV>, g, b,                                    \
               e.f.list_cap > 0 ? record_smem<DIM, RV, LV>(e.cfg.pair_block) : 0, st, e, \
               cur, dm, eos)
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
void launch_density_kt(const sphb_engine &e, int cur, uint32_t dm, int flags, cudaStream_t st)
{
    if constexpr (DIM == 2) {
        if (e.cfg.pair_mode == SPHB_PAIRS_TILED) {
            launch_density_tiled<KT>(e, cur, dm, flags, st);
            return;
        }
    }
    if (e.cfg.precision == SPHB_FP32C) launch_density_p<KT, DIM, true>(e, cur, dm, flags, st);
    else launch_density_p<KT, DIM, false>(e, cur, dm, flags, st);
}

}  // namespace sphb
