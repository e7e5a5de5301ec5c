// bp_fluid.cu -- position-based fluid passes (gather form, fixed neighbour order).
//
// Reference kernels (brasstower/kernel/fluid.cuh):
//   fluidLambda (:78-159)              -> k_lambda
//   fluidPosition (:161-228) + accDevArr_float3 (kernel/util.cuh:261-269)
//                                      -> k_deltap (gather, no atomics, epilogue fused)
//   fluidOmega (:231-279) + fluidNormal (:387-434)            -> k_post_a (one walk)
//   fluidVorticity (:281-336) + fluidAkinciTension (:436-488) -> k_post_b (one walk)
//   fluidXSph (:338-385)                                      -> k_post_c
//
// The reference scatters each pair's position correction to both particles
// with float atomics; here every particle gathers its own sum over the same
// pairs in a fixed order, so results are deterministic run to run.  The pair
// term for (k, j) is bit-identical to the reference's term for (j, k) up to
// sign, because the spiky gradient is odd in the difference vector.
#include <algorithm>

#include "bp_internal.h"
#include "bp_lists.cuh"

namespace bp {

constexpr int kScanThreads = kWalkThreads;  // scan kernels stage their neighbourhood (bp_walk.cuh)

// CTAs per SM the list-reading passes are compiled for.  The position pass
// loads each record's four positions and (lambda, mass) pairs before its four
// pair terms; at 4 CTAs (64 registers) that measured faster than at 5 (48
// registers, spilling), and than 5 CTAs with the pairs loaded per term
// (mixed scene 9.86 -> 9.68 ms per frame early, 15.40 -> 15.17 late).
#ifndef BP_DELTAP_MIN_BLOCKS
#define BP_DELTAP_MIN_BLOCKS 4
#endif
// Passes B and C load each record's neighbour data (|omega| and normal, or
// velocity) with the positions before the four pair terms; at 3 CTAs (80
// registers) that measured faster than at 4 (64, spilling) and than 4 CTAs
// with the data loaded per term (mixed scene 9.75 -> 9.62 ms per frame early,
// 15.24 -> 15.09 late).
#ifndef BP_POSTBC_MIN_BLOCKS
#define BP_POSTBC_MIN_BLOCKS 3
#endif

// Ends the Verlet list build of particle i (SimConsts::vl): its count, and
// the cell and position the list holds for (cell -1: no list, because it
// overflowed or the particle's column runs wrap around the table).
__device__ __forceinline__ void finish_verlet(const SimConsts &C, int i, float4 pi4, int cnt)
{
    const int3 c = cell_of(f3(pi4), C);
    const unsigned z0 = (unsigned)(c.z - 1) & C.mask, z2 = (unsigned)(c.z + 1) & C.mask;
    C.vl_count[i] = cnt;
    C.nl_pos[i] = pi4;
    C.nl_cell[i] = (cnt >= 0 && z0 < z2) ? cell_addr(c.x, c.y, c.z, C.D, C.mask) : -1;
}

// Reference mode (Q1): density sums only sorted indices j >= i; solid
// neighbours count x solid_scale; C = rho/rho0 - 1, clamped at 0 when Akinci
// is on; lambda = -C / lambda_den.  Textbook mode: all j, exact denominator.
//
// With C.nbr (neighbour lists on) the walk also records, for the position
// pass that reads the same positions, every j with r^2 <= h^2 in walk order
// (all j, also below i; solids too in reference mode, whose position pass
// gathers from fluid neighbours).  With C.vl_build it records the substep's
// Verlet lists instead: every j within h + skin.
template <bool Split, bool Stage>
__device__ __forceinline__ void k_lambda_tile(
    const SimConsts &C,
    const float4 *__restrict__ P,
    const float *__restrict__ mass,
    const int *__restrict__ off,
    float *__restrict__ lam,
    float *__restrict__ rho,
    int i0)
{
    StageShared &S = stage_shared();
    const int g = Stage ? stage_block(C, P, off, i0, S) : -1;
    const int t = i0 + threadIdx.x;  // the slot of the position pass's list
    if (t >= C.n) return;
    const int i = Stage ? t : walker_index(C, t);
    const float4 pi4 = P[i];
    const bool build = C.vl_build != 0;
    const bool rec = build || C.nbr != nullptr;
    // Slot lists: while the threads take class order (and no Verlet list can
    // stand in for a walk) the list holds class positions, and the position
    // pass gathers positions, masses and lambdas from the class-order copies.
    const bool slots = !Stage && C.nbr && !build && !C.vl && classes_on(C);
    const bool solid = phase_of(pi4) > 0;
    // (lambda, mass) for the position pass's gathers: by slot with slot
    // lists, by sorted index with lists of sorted indices
    auto put_lm = [&](float l) {
        if (slots) C.cls_lm[t] = make_float2(l, __ldg(mass + i));
        else if (C.lm && !build) C.lm[i] = make_float2(l, __ldg(mass + i));
    };
    if (solid) {  // solids carry lambda 0 (read by the position pass)
        lam[i] = 0.f;
        put_lm(0.f);
    }
    if (solid && (C.textbook || !rec)) {
        if (build) C.nl_cell[i] = -1;
        return;
    }
    const int sc = scene_index(C, i);
    const GridView v = grid_view(C, sc, off);
    const float rho0 = rest_density(C, sc);
    const float3 pi = f3(pi4);
    const float r2 = build ? C.nl_hs2 : C.h2;
    float density = 0.f;
    // Verlet lists are kept per particle, the position pass's lists per slot
    ListWriter list(build ? C.vl : C.nbr, build ? C.vl_cap : C.nbr_cap, C.n, build ? i : t);
    auto finish = [&]() {
        const int cnt = list.finish(i);
        if (build) finish_verlet(C, i, pi4, cnt);
        else C.nbr_count[t] = cnt;
    };
    auto record = [&](int &self) {  // entries: sorted indices, or class positions (slots)
        auto push = [&](int j, float4) {
            if (j == (slots ? t : i)) self = list.cnt;
            list.push(j);
        };
        auto test = [&](int, float4 pj) { return len2(pi - f3(pj)) <= r2; };
        // the walk planes hold the order this walk reads (class positions with
        // slots, sorted indices otherwise): the same hits in the same order
        const int planes = (Split && !Stage && !C.vl) ? walk_planes_order(C) : 0;
        if (planes == (slots ? 2 : 1)) {
            const int me = slots ? t : i;  // the particle's own entry
            record_walk_planes(planes, pi, r2, v, C, [&](int c0, unsigned bits) {
                const unsigned d = (unsigned)(me - c0);
                if (d < 32u && ((bits >> d) & 1u)) self = list.cnt + __popc(bits & ((1u << d) - 1u));
                list.push_bits(c0, bits);
            });
        } else if (slots) {  // the class walk walk_neighbors would take (no staging, no Verlet list), counted alike
            if (C.nl_stats) {
                atomicAdd(C.nl_stats + 1, 1u);
                atomicAdd(C.nl_stats + 4, 1u);
            }
            walk_classes<Split, true>(i, cell_of(pi, C), 0, v, C, test, push);
        } else {
            walk_neighbors<Split>(i, pi, 0, P, v, C, Stage ? &S : nullptr, g, test, push);
        }
        const int cnt = list.finish(slots ? t : i);
        C.nbr_count[t] = cnt;
        return cnt;
    };
    if (!C.textbook) {
        auto dens_m = [&](float mj, float4 pj) {
            const float ld = __fmul_rn(mj, poly6(C, len2(pi - f3(pj))));
            density = __fadd_rn(density, (phase_of(pj) < 0) ? ld : __fmul_rn(C.solid_scale, ld));
        };
        auto dens = [&](int j, float4 pj) { dens_m(__ldg(mass + j), pj); };
        auto test = [&](int, float4 pj) { return len2(pi - f3(pj)) <= r2; };
        if (C.nbr && !build) {
            // record first, then sum the density over the list's j >= i (the
            // mass gathers overlap there); an overflowed list walks again.
            // Where no column run wraps around the table the walk visits j in
            // ascending order, so the j >= i are the entries from i itself on.
            int self = kNoOwnEntry;
            const int cnt = record(self);
            if (solid) return;
            const int3 c = cell_of(pi, C);
            auto inner = [&](int a) {
                const unsigned u = (unsigned)a & v.mask;
                return u != 0u && u != v.mask;
            };
            const bool ascending = self != kNoOwnEntry && inner(c.x) && inner(c.y) && inner(c.z);
            const int first = ascending ? (self & ~3) : 0;
            if (cnt >= 0 && slots) {
                int e = first;  // entry index: ascending, the j >= i are the entries from self on
                for_each_in_list<false>(C.nbr, C.n, t, cnt, C.cls_pos, [&](int q, float4 pj) {
                    const bool upper = ascending ? e >= self : __ldg(C.cls_perm + q) >= i;
                    ++e;
                    if (upper) dens_m(__ldg(C.cls_mass + q), pj);
                }, first);
            } else if (cnt >= 0) {
                for_each_in_list<false>(C.nbr, C.n, t, cnt, P, [&](int j, float4 pj) {
                    if (j >= i) dens(j, pj);
                }, first);
            } else {
                walk_neighbors<Split>(i, pi, i, P, v, C, Stage ? &S : nullptr, g, test, dens);
            }
        } else {
            walk_neighbors<Split>(i, pi, rec ? 0 : i, P, v, C, Stage ? &S : nullptr, g, test,
                                  [&](int j, float4 pj) {
                                      if (rec) list.push(j);
                                      if (solid || j < i || (build && !(len2(pi - f3(pj)) <= C.h2))) return;
                                      dens(j, pj);
                                  });
            if (rec) finish();
        }
        if (solid) return;
        float c = density / rho0 - 1.0f;
        if (C.clamp_c) c = fmaxf(c, 0.0f);
        lam[i] = -c / C.lambda_den;
        put_lm(lam[i]);
    } else {
        const float inv_rho0 = inv_rest_density(C, sc);
        float sum_g2 = 0.f;
        float3 gi = make_float3(0.f, 0.f, 0.f);
        const float *mw = slots ? C.cls_mass : mass;  // indexed by the list's entries
        auto term = [&](int j, float4 pj) {
            const float3 diff = pi - f3(pj);
            const float d2 = len2(diff);
            const float mj = __ldg(mw + j);
            const float ld = __fmul_rn(mj, poly6(C, d2));
            density = __fadd_rn(density, (phase_of(pj) < 0) ? ld : __fmul_rn(C.solid_scale, ld));
            if (d2 > 0.f) {
                const float3 g = __fmul_rn(-mj, inv_rho0) * spiky_grad_r(C, diff, d2, rsqrtf(d2));
                sum_g2 = __fadd_rn(sum_g2, dot3(g, g));
                gi -= g;
            }
        };
        auto test = [&](int, float4 pj) { return len2(pi - f3(pj)) <= r2; };
        if (C.nbr && !build) {  // record first, then sum over the list (as above)
            int self = kNoOwnEntry;
            const int cnt = record(self);
            if (cnt >= 0) {
                for_each_in_list<false>(C.nbr, C.n, t, cnt, slots ? C.cls_pos : P, term);
            } else {
                mw = mass;  // the walk gives sorted indices
                walk_neighbors<Split>(i, pi, 0, P, v, C, Stage ? &S : nullptr, g, test, term);
            }
        } else {
            walk_neighbors<Split>(i, pi, 0, P, v, C, Stage ? &S : nullptr, g, test, [&](int j, float4 pj) {
                if (rec) list.push(j);
                if (build && !(len2(pi - f3(pj)) <= C.h2)) return;
                term(j, pj);
            });
            if (rec) finish();
        }
        float c = density / rho0 - 1.0f;
        if (C.clamp_c) c = fmaxf(c, 0.0f);
        sum_g2 += dot3(gi, gi);
        lam[i] = -c / (sum_g2 + C.relaxation);
        put_lm(lam[i]);
    }
    rho[i] = density;
    if (slots) C.cls_rho[t] = density;
}

template <bool Split, bool Stage, bool Persist = false>
__global__ void __launch_bounds__(kScanThreads, BP_SCAN_MIN_BLOCKS) k_lambda(
    SimConsts C,
    const float4 *__restrict__ P,
    const float *__restrict__ mass,
    const int *__restrict__ off,
    float *__restrict__ lam,
    float *__restrict__ rho)
{
    // one tile of blockDim.x particles per CTA, or, persistent (an unstaged
    // launch of at most one resident wave: SimConsts::scan_persist), every
    // gridDim.x-th tile from blockIdx.x on
    if constexpr (Persist) {
        for (int i0 = blockIdx.x * blockDim.x; i0 < C.n; i0 += gridDim.x * blockDim.x)
            k_lambda_tile<Split, Stage>(C, P, mass, off, lam, rho, i0);
    } else {
        k_lambda_tile<Split, Stage>(C, P, mass, off, lam, rho, blockIdx.x * blockDim.x);
    }
}

// Kernels with a split walk (test, then body over the hits) and a fused one.
// Kernels instantiated for split / fused walks and staged / unstaged CTAs
// (an unstaged instantiation carries none of the staging code or registers).
// Persistent launches (SimConsts::scan_persist) exist for the split,
// unstaged instantiation, the one the autotuner keeps almost everywhere.
#define BP_LAUNCH_SPLIT(kernel, st, ...)                                                              \
    do {                                                                                              \
        const size_t smem_ = stage_bytes(C);                                                          \
        if (C.split && C.stage) launch_scan(kernel<true, true>, C, smem_, st, __VA_ARGS__);           \
        else if (C.split && C.scan_persist) launch_scan(kernel<true, false, true>, C, smem_, st, __VA_ARGS__); \
        else if (C.split) launch_scan(kernel<true, false>, C, smem_, st, __VA_ARGS__);                \
        else if (C.stage) launch_scan(kernel<false, true>, C, smem_, st, __VA_ARGS__);                \
        else launch_scan(kernel<false, false>, C, smem_, st, __VA_ARGS__);                            \
    } while (0)

void launch_lambda(cudaStream_t st, const SimConsts &C, const float4 *P, const float *mass, const int *off,
                   float *lam, float *rho, LaunchLog *L)
{
    if (C.n <= 0) return;
    BP_LAUNCH_SPLIT(k_lambda, st, C, P, mass, off, lam, rho);
    L->done(__func__);
}

// ---- the passes over the substep lists (bp_lists.cuh) ----

// Writes a fluid particle's density and lambda, and their copies.
__device__ __forceinline__ void finish_lambda(const SimConsts &C, bool slots, int i, int t, float density, float rho0,
                                              float den, const float *__restrict__ mass, float *__restrict__ lam,
                                              float *__restrict__ rho)
{
    float c = density / rho0 - 1.0f;
    if (C.clamp_c) c = fmaxf(c, 0.0f);
    const float l = -c / den;
    lam[i] = l;
    if (slots) {
        C.cls_lm[t] = make_float2(l, __ldg(mass + i));
        C.cls_rho[t] = density;
    } else {
        C.lm[i] = make_float2(l, __ldg(mass + i));
    }
    rho[i] = density;
}

// A solid's lambda, 0, and its pair for the position pass's gathers.  Later
// passes of the substep leave solids out, so the pair goes to both orders: the
// classes may close in between (k_class_refresh), and the lists then hold
// sorted indices.
__device__ __forceinline__ void record_solid(const SimConsts &C, bool slots, int i, int t,
                                             const float *__restrict__ mass, float *__restrict__ lam)
{
    const float2 lm = make_float2(0.f, __ldg(mass + i));
    lam[i] = 0.f;
    C.lm[i] = lm;
    if (slots) C.cls_lm[t] = lm;
}

// Records slot t's contact partners (SimConsts::cl_list) from its list just
// recorded.
__device__ __forceinline__ void record_contacts(const SimConsts &C, const float4 *__restrict__ P, bool slots, int t,
                                                int i, float4 pi4, int3 c, const GridView &v, int packed, float touch2)
{
    const int phi = phase_of(pi4);
    const int addr = cell_addr(c.x, c.y, c.z, v.D, v.mask);
    int n = 0;
    if (packed < 0) {
        n = kContactCap + 1;
    } else if (phi > 0 || !C.cl_near || ((__ldg(C.cl_near + (addr >> 6)) >> (addr & 63)) & 1ull)) {
        auto none = [](int) { return 0; };
        for_each_padded<false>(C.nbr, C.n, t, packed & 0xffff, slots ? C.cls_pos : P, none, [&](int q, float4 pj4, int) {
            const int phj = phase_of(pj4);  // the own entry: the same phase
            if (phi == phj || !(phi > 0 || phj > 0) || !(len2(f3(pi4) - f3(pj4)) <= touch2)) return;
            if (n < kContactCap) C.cl_list[(size_t)n * C.n + t] = slots ? __ldg(C.cls_perm + q) : q;
            ++n;
        });
    }
    C.cl_count[t] = n <= kContactCap ? n : -1;
}

// The density (and, in textbook mode, the denominator) of fluid particle i of
// slot t over its list (packed: what nbr_count holds), as k_lambda sums it over
// the same pairs in the same order.  ReadOnly: the calling thread did not write
// the list.  pairs (textbook mode): grows by the entries within h.
template <bool ReadOnly>
__device__ __forceinline__ void lambda_over_list(const SimConsts &C, const float4 *__restrict__ P,
                                                 const float *__restrict__ mass, float *__restrict__ lam,
                                                 float *__restrict__ rho, bool slots, int i, int t, float4 pi4, int sc,
                                                 int3 c, const GridView &v, int packed, int &pairs)
{
    const float3 pi = f3(pi4);
    const int cnt = packed & 0xffff, self = packed >> 16;
    const float4 *__restrict__ src = slots ? C.cls_pos : P;
    const float *__restrict__ ms = slots ? C.cls_mass : mass;
    const float rho0 = rest_density(C, sc);
    float density = 0.f, den = C.lambda_den;
    auto fetch = [&](int j) { return __ldg(ms + j); };
    if (!C.textbook) {
        auto add = [&](float mj, float4 pj, float d2) {
            const float ld = __fmul_rn(mj, poly6(C, d2));
            density = __fadd_rn(density, (phase_of(pj) < 0) ? ld : __fmul_rn(C.solid_scale, ld));
        };
        if (packed >= 0) {
            // j >= i: where no column run wraps around the table the walk is
            // in ascending j, so these are the entries from the own one on
            auto inner = [&](int a) {
                const unsigned u = (unsigned)a & v.mask;
                return u != 0u && u != v.mask;
            };
            const bool ascending = self != kNoOwnEntry && inner(c.x) && inner(c.y) && inner(c.z);
            int e = ascending ? (self & ~3) : 0;
            const int first = e;
            for_each_padded<ReadOnly>(C.nbr, C.n, t, cnt, src, fetch, [&](int j, float4 pj, float mj) {
                const float d2 = len2(pi - f3(pj));
                bool take = d2 <= C.h2;
                if (ascending) take = take && (unsigned)(e - self) < (unsigned)(cnt - self);
                else take = take && e < cnt && (slots ? __ldg(C.cls_perm + j) : j) >= i;
                ++e;
                if (take) add(mj, pj, d2);
            }, first);
        } else {
            auto test = [&](int, float4 pj) { return len2(pi - f3(pj)) <= C.h2; };
            walk_neighbors<true>(i, pi, i, P, v, C, nullptr, -1, test,
                                 [&](int j, float4 pj) { add(__ldg(mass + j), pj, len2(pi - f3(pj))); });
        }
    } else {
        const float inv_rho0 = inv_rest_density(C, sc);
        float sum_g2 = 0.f;
        float3 gi = make_float3(0.f, 0.f, 0.f);
        auto term = [&](float mj, float4 pj) {
            const float3 diff = pi - f3(pj);
            const float d2 = len2(diff);
            if (!(d2 <= C.h2)) return;
            const float ld = __fmul_rn(mj, poly6(C, d2));
            density = __fadd_rn(density, (phase_of(pj) < 0) ? ld : __fmul_rn(C.solid_scale, ld));
            if (d2 > 0.f) {
                const float3 g = __fmul_rn(-mj, inv_rho0) * spiky_grad_r(C, diff, d2, rsqrtf(d2));
                sum_g2 = __fadd_rn(sum_g2, dot3(g, g));
                gi -= g;
            }
        };
        if (packed >= 0) {
            int e = 0;
            for_each_padded<ReadOnly>(C.nbr, C.n, t, cnt, src, fetch, [&](int, float4 pj, float mj) {
                // (counted here, the terms' distances are free of the branch: 85.8 ->
                // 79.6 us a reading pass of 829,440 particles)
                pairs += len2(pi - f3(pj)) <= C.h2 ? 1 : 0;
                if (e++ < cnt) term(mj, pj);
            });
        } else {
            auto test = [&](int, float4 pj) { return len2(pi - f3(pj)) <= C.h2; };
            walk_neighbors<true>(i, pi, 0, P, v, C, nullptr, -1, test,
                                 [&](int j, float4 pj) { term(__ldg(mass + j), pj); });
        }
        sum_g2 += dot3(gi, gi);
        den = sum_g2 + C.relaxation;
    }
    finish_lambda(C, slots, i, t, density, rho0, den, mass, lam, rho);
}

// The lambda pass over the substep lists: the density (and, in textbook mode,
// the denominator) of k_lambda, from the same pairs in the same order.
// What bounds it: a list read is latency-bound on its gathers, like k_deltap;
// the recording walk is issue-bound, like k_lambda.
// Walks: the substeps may be in walk mode; the recording pass then counts, over
// every kSampleBlocks-th CTA, the entries it sums over and the pairs among them
// (choose_mode).  Instances of their own: the mode costs the reading one 4 %.
constexpr int kSampleBlocks = 64;
template <ListPass Pass, bool Walks>
__device__ __forceinline__ void lambda_substep_list(const SimConsts &C, const float4 *__restrict__ P,
                                                    const float *__restrict__ mass, const int *__restrict__ off,
                                                    float *__restrict__ lam, float *__restrict__ rho, int t)
{
    const bool walking = Walks && walk_mode(C);  // loaded along with the particle
    const bool slots = classes_on(C);
    const int i = slots ? __ldg(C.cls_perm + t) : t;
    const float4 pi4 = slots ? C.cls_pos[t] : P[i];
    const float3 pi = f3(pi4);
    const bool solid = phase_of(pi4) > 0;
    if (Pass == kRecordLists) {
        C.sl_pos[i] = pi4;
        if (solid && C.sl_fluid) record_solid(C, slots, i, t, mass, lam);
    }
    // textbook mode: no pass but the contacts moves a solid by its neighbours
    if (solid && C.textbook && !(Pass == kRecordLists && C.cl_list)) return;
    const int sc = scene_index(C, i);
    const GridView v = grid_view(C, sc, off);
    const int3 c = cell_of(pi, C);
    int packed;
    if (Pass == kReadLists && walking) {
        note_substep_list(C, t, i, pi, c, v);
        packed = record_substep_list(C, P, slots, t, i, pi, c, C.h2, v);
        C.nbr_count[t] = packed;
    } else if (Pass == kReadLists) {
        if (!reads_substep_list(C, t, i, pi, c, v) || solid) return;
        packed = __ldg(C.nbr_count + t);
    } else {
        const float skin = substep_skin(C), touch = 2.0f * C.radius + skin;
        const float reach = fmaxf(C.sl_fluid ? (walking ? C.h : C.h + skin) : 0.f, C.cl_list ? touch : 0.f);
        packed = record_substep_list(C, P, slots, t, i, pi, c, __fmul_rn(reach, reach), v);
        const bool fits = packed >= 0;
        if (C.cl_list) record_contacts(C, P, slots, t, i, pi4, c, v, packed, __fmul_rn(touch, touch));
        // the neighbours within h alone may still fit; later passes then walk
        if (!fits && C.sl_fluid) packed = record_substep_list(C, P, slots, t, i, pi, c, C.h2, v);
        C.nbr_count[t] = packed;
        C.sl_cell[t] = (fits && near_stored_cell(C, i, c, v)) ? v.base + cell_addr(c.x, c.y, c.z, v.D, v.mask) : kListNone;
        if (!C.sl_fluid) return;
    }
    if (solid) return;
    int pairs = 0;
    // a pass that may walk reads its lists past the read-only path
    lambda_over_list<Pass == kReadLists && !Walks>(C, P, mass, lam, rho, slots, i, t, pi4, sc, c, v, packed, pairs);
    if (Pass == kRecordLists && Walks && blockIdx.x % kSampleBlocks == 0 && packed >= 0) {
        const int found[3] = {pairs, packed & 0xffff, walk_candidates(C, slots, i, c, v)};
        const unsigned m = __activemask();
        const bool first = (threadIdx.x & 31) == __ffs(m) - 1;
        if (first) atomicAdd(C.sl_count + kSlSample, __popc(m));
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int sum = __reduce_add_sync(m, found[k]);
            if (first) atomicAdd(C.sl_count + kSlPairs + k, sum);
        }
    }
}

template <ListPass Pass, bool Walks>
__global__ void __launch_bounds__(kScanThreads, BP_SCAN_MIN_BLOCKS) k_lambda_lists(
    SimConsts C, const float4 *__restrict__ P, const float *__restrict__ mass, const int *__restrict__ off,
    float *__restrict__ lam, float *__restrict__ rho)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) {
        C.sl_count[C.sl_pass ^ 1] = 0;  // the next pass's queue
        if (Pass == kRecordLists) {
            C.sl_count[C.sl_pass] = 0;
            C.sl_count[kSlDisplaced] = C.sl_count[kSlWalks] = C.sl_count[kSlContactWalks] = 0;
            C.sl_count[kSlMoved] = C.cls_perm ? *C.cls_moved : 0;
        }
    }
    if (t < C.n) lambda_substep_list<Pass, Walks>(C, P, mass, off, lam, rho, t);
}

// The queued particles' lambda pass, a warp per particle: walks the
// cells, leaves the neighbours within h in the list for this iteration's
// position pass, and adds the pair terms, computed a candidate per lane, in
// walk order.
constexpr int kQueueThreads = 128;
__global__ void __launch_bounds__(kQueueThreads) k_lambda_queued(SimConsts C, const float4 *__restrict__ P,
                                                                const float *__restrict__ mass,
                                                                const int *__restrict__ off, float *__restrict__ lam,
                                                                float *__restrict__ rho)
{
    __shared__ WarpRows rows[kQueueThreads / 32];
    __shared__ WarpHits hits[kQueueThreads / 32];
    const int lane = threadIdx.x & 31;
    const int queued = C.sl_count[C.sl_pass];
    adapt_skin(C);
    const bool slots = classes_on(C);
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) / 32; k < queued; k += gridDim.x * blockDim.x / 32) {
        const int t = C.sl_queue[k];
        const int i = slots ? __ldg(C.cls_perm + t) : t;
        const float4 pi4 = slots ? C.cls_pos[t] : P[i];
        const float3 pi = f3(pi4);
        const bool solid = phase_of(pi4) > 0;  // its list only (reference mode)
        const int sc = scene_index(C, i);
        const GridView v = grid_view(C, sc, off);
        const float inv_rho0 = inv_rest_density(C, sc);
        if (C.nl_stats && slots && lane == 0) atomicAdd(C.nl_stats + 4, 1u);
        float acc = 0.f;  // lane 0: the density; textbook, lanes 1..4: sum of g^2, -sum of g
        int self = kNoOwnEntry;
        const int me = slots ? t : i;
        auto test = [&](int, float4 pj) { return len2(pi - f3(pj)) <= C.h2; };
        auto batch = [&](int k0, int n, int q, float4 pj) {
            const bool in = lane < n;
            if (in) put_entry(C, t, k0 + lane, q);
            const unsigned own = __ballot_sync(kWarp, in && q == me);
            if (own) self = k0 + __ffs(own) - 1;
            if (solid) return;
            bool take = in;
            float value[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
            if (in) {
                const int j = slots ? __ldg(C.cls_perm + q) : q;
                const float mj = __ldg((slots ? C.cls_mass : mass) + q);
                const float3 diff = pi - f3(pj);
                const float d2 = len2(diff);
                take = C.textbook || j >= i;
                value[0] = __fmul_rn(mj, poly6(C, d2));
                if (phase_of(pj) >= 0) value[0] = __fmul_rn(C.solid_scale, value[0]);
                if (C.textbook && d2 > 0.f) {  // the pair at r = 0 adds zeros
                    const float3 g = __fmul_rn(-mj, inv_rho0) * spiky_grad_r(C, diff, d2, rsqrtf(d2));
                    value[1] = dot3(g, g);
                    value[2] = -g.x;
                    value[3] = -g.y;
                    value[4] = -g.z;
                }
            }
            warp_add(rows[threadIdx.x >> 5], __ballot_sync(kWarp, take), value, 1.f, acc);
        };
        const int cnt = warp_neighbors(C, slots, cell_of(pi, C), P, v, hits[threadIdx.x >> 5], test, batch);
        warp_pad(C, t, cnt, slots ? t : i);
        const float sum_g2 = __shfl_sync(kWarp, acc, 1);
        const float3 gi = make_float3(__shfl_sync(kWarp, acc, 2), __shfl_sync(kWarp, acc, 3), __shfl_sync(kWarp, acc, 4));
        if (lane != 0) continue;
        C.nbr_count[t] = cnt <= C.nbr_cap ? cnt | (self << 16) : -1;
        if (solid) continue;
        finish_lambda(C, slots, i, t, acc, rest_density(C, sc),
                      C.textbook ? (sum_g2 + dot3(gi, gi)) + C.relaxation : C.lambda_den, mass, lam, rho);
    }
}

// Moves particle k by its summed corrections, then the pass's epilogue.
__device__ __forceinline__ void finish_deltap(const SimConsts &C, const DeltaArgs &a, int sc, int k, float4 pk4,
                                              float3 sum)
{
    float3 p = f3(pk4) + sum * inv_rest_density(C, sc);
    if (a.epilogue == 1) {
        plane_collide(C, sc, f3(a.Xs[k]), p);
    } else if (a.epilogue == 2) {  // updateVelocity + updatePositions (PS:71-81, 121-137)
        const float4 xs = a.Xs[k];
        const float3 v = (p - f3(xs)) * C.inv_dt;
        a.Xc[k] = make_float4(p.x, p.y, p.z, xs.w);
        a.Vc[k] = make_float4(v.x, v.y, v.z, pk4.w);
        a.orig_c[k] = a.orig_s[k];
    }
    a.Pout[k] = make_float4(p.x, p.y, p.z, pk4.w);
    if (C.sl_planes && walk_mode(C)) put_planes(C.sl_planes, C.walk_stride, k, make_float4(p.x, p.y, p.z, pk4.w));
    track_displacement(C, k, p, true);
}

// Position correction.  Reference mode: the pair (a, b), a < b, contributes
// when a is a fluid particle (only fluid threads run fluidPosition and they
// only visit b > a), to both ends.  In gather form particle k includes j when
// the lower-indexed of (k, j) is fluid.  Textbook mode: fluid k gathers over
// every neighbour; solids do not move.  With C.nbr the neighbours come from
// the lists k_lambda recorded at the same positions (r^2 <= h^2, walk order);
// particles whose list overflowed walk their cells.
template <bool Split, bool Stage>
__device__ __forceinline__ void k_deltap_tile(
    const SimConsts &C,
    DeltaArgs a,
    int i0)
{
    StageShared &S = stage_shared();
    const int t = i0 + threadIdx.x;  // the slot of k's list (k_lambda)
    const bool valid = t < C.n;
    const int k = (Stage || !valid) ? t : walker_index(C, t);
    const float4 pk4 = valid ? a.P[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int phk = phase_of(pk4);
    const bool moves = valid && !(C.textbook && phk > 0);
    int listed = (moves && C.nbr) ? __ldg(C.nbr_count + t) : -1;
    const bool walk = moves && listed < 0;
    listed &= 0xffff;  // substep lists: above it, the own entry's index
    // substep lists also hold entries past h (the test changes nothing for
    // lists of the neighbours within h); r = 0 excludes k itself
    auto near = [&](float d2) { return d2 > 0.f && d2 <= C.h2; };
    const int g = (Stage && __syncthreads_or(walk)) ? stage_block(C, a.P, a.off, i0, S) : -1;
    if (!valid) return;
    const float3 pk = f3(pk4);
    const int sc = scene_index(C, k);
    float3 sum = make_float3(0.f, 0.f, 0.f);
    if (moves) {
        const float lk = a.lam[k];
        // adds the pair term where ok; the rest of it has no condition
        auto pair_at = [&](bool ok, float3 diff, float d2, float lj, float mj) {
            float sl = __fadd_rn(lk, lj);
            if (C.scorr_on)
                sl = __fsub_rn(sl, __fmul_rn(C.scorr_k, ipowf(__fmul_rn(poly6(C, d2), C.scorr_inv_wq), C.scorr_ni)));
            float3 delta = sl * spiky_grad_r(C, diff, d2, rsqrtf(d2));
            if (C.delta_clamp > 0.f) {  // per-pair clamp; the length is only needed past it
                const float l2 = len2(delta);
                if (ok && !(l2 < C.delta_clamp2)) delta = delta * __fmul_rn(C.delta_clamp, rsqrtf(l2));
            }
            if (ok) sum = fma3(mj, delta, sum);
        };
        auto pair = [&](float4 pj4, float lj, float mj) {
            const float3 diff = pk - f3(pj4);
            pair_at(true, diff, len2(diff), lj, mj);
        };
        auto body = [&](int j, float4 pj4) {
            if (!C.textbook && !((j > k) ? (phk < 0) : (phase_of(pj4) < 0))) return;
            pair(pj4, __ldg(a.lam + j), __ldg(a.mass + j));
        };
        // slot lists (k_lambda) hold class positions q: the pair's data come
        // from the class-order copies, the sorted index only where one of the
        // two is a solid (the fluid-fluid pairs pass the rule either way)
        const bool slots = !Stage && C.nbr && !C.vl && classes_on(C);
        // each entry's (lambda, mass) loads with its position, before the
        // four pair terms of a record
        if (!walk && slots) {
            auto fetch = [&](int q) { return __ldg(C.cls_lm + q); };
            for_each_padded(C.nbr, C.n, t, listed, C.cls_pos, fetch, [&](int q, float4 pj4, float2 lm) {
                const float3 diff = pk - f3(pj4);
                const float d2 = len2(diff);
                bool ok = near(d2);
                const bool fj = phase_of(pj4) < 0;
                if (!C.textbook && !(phk < 0 && fj)) ok = ok && ((__ldg(C.cls_perm + q) > k) ? (phk < 0) : fj);
                pair_at(ok, diff, d2, lm.x, lm.y);
            });
        } else if (!walk && C.lm) {
            auto fetch = [&](int j) { return __ldg(C.lm + j); };
            for_each_padded(C.nbr, C.n, t, listed, a.P, fetch, [&](int j, float4 pj4, float2 lm) {
                const float3 diff = pk - f3(pj4);
                const float d2 = len2(diff);
                bool ok = near(d2);
                if (!C.textbook) ok = ok && ((j > k) ? (phk < 0) : (phase_of(pj4) < 0));
                pair_at(ok, diff, d2, lm.x, lm.y);
            });
        } else if (!walk) {
            auto listed_body = [&](int j, float4 pj4) {
                if (near(len2(pk - f3(pj4)))) body(j, pj4);
            };
            for_each_in_list(C.nbr, C.n, t, listed, a.P, listed_body);
        } else {
            walk_neighbors<Split>(
                k, pk, 0, a.P, grid_view(C, sc, a.off), C, Stage ? &S : nullptr, g,
                [&](int, float4 pj4) {  // r = 0 excludes k itself
                    const float d2 = len2(pk - f3(pj4));
                    return d2 <= C.h2 && d2 > 0.f;
                },
                body);
        }
    }
    finish_deltap(C, a, sc, k, pk4, sum);
}

template <bool Split, bool Stage, bool Persist = false>
__global__ void __launch_bounds__(kScanThreads, BP_DELTAP_MIN_BLOCKS) k_deltap(
    SimConsts C,
    DeltaArgs a)
{
    // one tile of blockDim.x particles per CTA, or, persistent (an unstaged
    // launch of at most one resident wave: SimConsts::scan_persist), every
    // gridDim.x-th tile from blockIdx.x on
    if constexpr (Persist) {
        for (int i0 = blockIdx.x * blockDim.x; i0 < C.n; i0 += gridDim.x * blockDim.x)
            k_deltap_tile<Split, Stage>(C, a, i0);
    } else {
        k_deltap_tile<Split, Stage>(C, a, blockIdx.x * blockDim.x);
    }
}

// The post passes keep class positions in their lists (SimConsts::cls_post):
// pass A records them and every pass reads its neighbours' data from the
// class-order copies, as k_lambda and k_deltap do.
__device__ __forceinline__ bool post_slots(const SimConsts &C, bool stage)
{
    return !stage && C.cls_post && C.nbr && C.nbr_count && !C.vl && classes_on(C);
}

// Pass A: vorticity omega_i (fluidOmega) and Akinci normal n_i (fluidNormal)
// in one walk over same-phase neighbours with 0 < r^2 <= h^2.
// Om[i] = (omega, |omega|); Nm[i] = (h * n, rho_i).
template <bool Split, bool Stage>
__device__ __forceinline__ void k_post_a_tile(
    const SimConsts &C,
    const float4 *__restrict__ P,
    const float4 *__restrict__ V,
    const float *__restrict__ rho,
    const int *__restrict__ off,
    float4 *__restrict__ Om,
    float4 *__restrict__ Nm,
    int i0)
{
    StageShared &S = stage_shared();
    const int g = Stage ? stage_block(C, P, off, i0, S) : -1;
    const int t = i0 + threadIdx.x;  // the slot of the list passes B and C read
    if (t >= C.n) return;
    const int i = Stage ? t : walker_index(C, t);
    const float4 pi4 = P[i];
    const int phi = phase_of(pi4);
    if (phi >= 0) return;
    const float3 pi = f3(pi4);
    const float3 vi = f3(V[i]);
    float3 om = make_float3(0.f, 0.f, 0.f), nn = make_float3(0.f, 0.f, 0.f);
    const bool want_om = C.use_vort, want_n = C.use_akinci;
    const bool slots = post_slots(C, Stage);
    auto term_at = [&](const float4 *__restrict__ Vp, const float *__restrict__ rp, int j, float4 pj4) {
        const float3 diff = pi - f3(pj4);
        const float d2 = len2(diff);
        if (!(d2 > 0.f)) return;
        const float3 g = spiky_grad_r(C, diff, d2, rsqrtf(d2));
        if (want_om) om += cross3(f3(Vp[j]) - vi, g);
        if (want_n) nn = fma3(__frcp_rn(__ldg(rp + j)), g, nn);
    };
    auto term = [&](int j, float4 pj4) { term_at(V, rho, j, pj4); };
    const GridView v = grid_view(C, scene_index(C, i), off);
    auto test = [&](int, float4 pj4) { return len2(pi - f3(pj4)) <= C.h2; };
    // The walk takes the passes' common neighbours (r = 0 included, as pass C
    // wants them).  With lists on it only records them (for passes B and C as
    // well), and the terms are then summed over the list four neighbours at a
    // time, so their velocity and density gathers overlap; a list that
    // overflowed is summed by walking again.
    int cnt = -1;
    if (C.nbr) {
        ListWriter list(C.nbr, C.nbr_cap, C.n, t);
        // the walk planes hold the order this walk reads (class positions with
        // slots, sorted indices otherwise): the same hits in the same order,
        // each chunk's kept where the phase plane matches and not the own entry
        const int planes = (Split && !Stage && !C.vl) ? walk_planes_order(C) : 0;
        if (planes == (slots ? 2 : 1)) {
            const int *__restrict__ W = reinterpret_cast<const int *>(C.walk_xyz) + 3 * (size_t)C.walk_stride;
            const int me = slots ? t : i;
            record_walk_planes(planes, pi, C.h2, v, C, [&](int c0, unsigned bits) {
                const unsigned d = (unsigned)(me - c0);
                if (d < 32u) bits &= ~(1u << d);
                unsigned same = 0u;
                for (unsigned quads = bits; quads;) {  // the phases of the quads holding hits
                    const int q4 = (__ffs(quads) - 1) & ~3;
                    const int4 w = __ldg(reinterpret_cast<const int4 *>(W + c0 + q4));
                    same |= ((w.x == phi ? 1u : 0u) | (w.y == phi ? 2u : 0u) | (w.z == phi ? 4u : 0u) |
                             (w.w == phi ? 8u : 0u))
                            << q4;
                    quads &= ~(0xfu << q4);
                }
                list.push_bits(c0, bits & same);
            });
        } else if (slots) {  // the class walk walk_neighbors would take, recording class positions
            if (C.nl_stats) {
                atomicAdd(C.nl_stats + 1, 1u);
                atomicAdd(C.nl_stats + 4, 1u);
            }
            auto push = [&](int q, float4 pj4) {
                if (q != t && phase_of(pj4) == phi) list.push(q);
            };
            walk_classes<Split, true>(i, cell_of(pi, C), 0, v, C, test, push);
        } else {
            walk_neighbors<Split>(i, pi, 0, P, v, C, Stage ? &S : nullptr, g, test, [&](int j, float4 pj4) {
                if (j != i && phase_of(pj4) == phi) list.push(j);
            });
        }
        cnt = list.finish(slots ? t : i);
        C.nbr_count[t] = cnt;
        // the records just written come back through the coherent path (plain loads)
        if (cnt >= 0 && slots)
            for_each_in_list<false>(C.nbr, C.n, t, cnt, C.cls_pos,
                                    [&](int q, float4 pj4) { term_at(C.cls_vel, C.cls_rho, q, pj4); });
        else if (cnt >= 0)
            for_each_in_list<false>(C.nbr, C.n, t, cnt, P, term);
    }
    if (cnt < 0)
        walk_neighbors<Split>(i, pi, 0, P, v, C, Stage ? &S : nullptr, g, test, [&](int j, float4 pj4) {
            if (j != i && phase_of(pj4) == phi) term(j, pj4);
        });
    const float4 om4 = make_float4(om.x, om.y, om.z, len3(om));
    const float3 n = C.h * nn;
    const float4 nm4 = make_float4(n.x, n.y, n.z, rho[i]);
    Om[i] = om4;
    Nm[i] = nm4;
    if (slots) {
        C.cls_om[t] = om4;
        C.cls_nm[t] = nm4;
    }
}

template <bool Split, bool Stage, bool Persist = false>
__global__ void __launch_bounds__(kScanThreads, BP_SCAN_MIN_BLOCKS) k_post_a(
    SimConsts C,
    const float4 *__restrict__ P,
    const float4 *__restrict__ V,
    const float *__restrict__ rho,
    const int *__restrict__ off,
    float4 *__restrict__ Om,
    float4 *__restrict__ Nm)
{
    // one tile of blockDim.x particles per CTA, or, persistent (an unstaged
    // launch of at most one resident wave: SimConsts::scan_persist), every
    // gridDim.x-th tile from blockIdx.x on
    if constexpr (Persist) {
        for (int i0 = blockIdx.x * blockDim.x; i0 < C.n; i0 += gridDim.x * blockDim.x)
            k_post_a_tile<Split, Stage>(C, P, V, rho, off, Om, Nm, i0);
    } else {
        k_post_a_tile<Split, Stage>(C, P, V, rho, off, Om, Nm, blockIdx.x * blockDim.x);
    }
}

// Passes B and C: the number of recorded neighbours of particle i (its list
// in slot t, k_post_a), or kWalkCells when it must walk its cells (no lists,
// or they overflowed).  Solids and indices past the end need neither (0).
constexpr int kWalkCells = -1;
__device__ __forceinline__ int post_list_count(const SimConsts &C, const float4 *__restrict__ P, int i, int t)
{
    if (i >= C.n || phase_of(P[i]) >= 0) return 0;
    if (!C.nbr || !C.nbr_count) return kWalkCells;
    const int cnt = __ldg(C.nbr_count + t);
    return cnt >= 0 ? cnt & 0xffff : kWalkCells;  // substep lists: above it, the own entry's index
}

// Particle i's velocity from its pass B sums.
__device__ __forceinline__ void finish_post_b(const SimConsts &C, bool slots, int i, int t, float4 vi4, float3 eta,
                                              float3 ft, const float4 *__restrict__ Om, float4 *__restrict__ Vout)
{
    float3 v = f3(vi4);
    if (C.use_vort && len2(eta) > 1e-3f) {
        const float inv = 1.0f / sqrtf(dot3(eta, eta));
        const float3 nrm = eta * inv;
        v += (C.vort_eps * cross3(nrm, f3(Om[i]))) * C.dt;
    }
    if (C.use_akinci) v = v + ft * C.dt;
    const float4 v4 = make_float4(v.x, v.y, v.z, vi4.w);
    Vout[i] = v4;
    if (slots) C.cls_vb[t] = v4;  // pass C's neighbour velocities
}

// Pass B: vorticity confinement (fluidVorticity) then Akinci tension
// (fluidAkinciTension), both on the same neighbours.  v' = v + eps (N x w) dt,
// v'' = v' + F dt, exactly the reference's sequence (in-place update followed
// by newVelocities = velocities + F dt).  Solids pass through.
template <bool Split, bool Stage>
__device__ __forceinline__ void k_post_b_tile(
    const SimConsts &C,
    const float4 *__restrict__ P,
    const float4 *__restrict__ V,
    const float4 *__restrict__ Om,
    const float4 *__restrict__ Nm,
    const int *__restrict__ off,
    float4 *__restrict__ Vout,
    int i0)
{
    StageShared &S = stage_shared();
    const int t = i0 + threadIdx.x;
    const int i = (Stage || t >= C.n) ? t : walker_index(C, t);
    const int cnt = post_list_count(C, P, i, t);
    const int g = (Stage && __syncthreads_or(cnt == kWalkCells)) ? stage_block(C, P, off, i0, S) : -1;
    if (i >= C.n) return;
    const float4 pi4 = P[i];
    const float4 vi4 = V[i];
    const int phi = phase_of(pi4);
    if (phi >= 0) {
        Vout[i] = vi4;
        return;
    }
    const int sc = scene_index(C, i);
    const float two_rho0 = 2.0f * rest_density(C, sc);
    const float3 pi = f3(pi4);
    const float4 ni4 = Nm[i];
    const float3 ni = f3(ni4);
    const float rhoi = ni4.w;
    float3 eta = make_float3(0.f, 0.f, 0.f), ft = make_float3(0.f, 0.f, 0.f);
    const bool want_v = C.use_vort, want_t = C.use_akinci;
    const bool slots = post_slots(C, Stage);
    // a neighbour's |omega| and (h n, rho), as the pair terms read them
    struct Nb {
        float om;
        float4 nm;
    };
    auto fetch_at = [&](const float4 *__restrict__ Omp, const float4 *__restrict__ Nmp, int j) {
        Nb r;
        r.om = want_v ? Omp[j].w : 0.f;
        r.nm = want_t ? Nmp[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        return r;
    };
    auto pair_terms = [&](float4 pj4, const Nb &nb) {
        const float3 diff = pi - f3(pj4);
        const float d2 = len2(diff);
        // the last two hold for the lists pass A records, not for substep lists
        const bool ok = d2 > 0.f && d2 <= C.h2 && phase_of(pj4) == phi;
        const float inv_r = rsqrtf(d2);
        const float3 g = spiky_grad_r(C, diff, d2, inv_r);
        if (ok && want_v) eta = fma3(nb.om, g, eta);
        if (ok && want_t) {
            const float4 nj4 = nb.nm;
            const float dist = __fmul_rn(d2, inv_r);
            const float3 fco = __fmul_rn(__fmul_rn(-C.tension, akinci_spline(C, dist)), inv_r) * diff;
            const float3 fcu = (-C.tension) * (ni - f3(nj4));
            const float kij = __fmul_rn(two_rho0, __frcp_rn(__fadd_rn(rhoi, nj4.w)));
            ft = fma3(kij, fco + fcu, ft);
        }
    };
    auto body = [&](int j, float4 pj4) { pair_terms(pj4, fetch_at(Om, Nm, j)); };
    // each entry's omega and normal load with its position, before the four
    // pair terms of a record
    auto listed = [&](int, float4 pj4, const Nb &nb) { pair_terms(pj4, nb); };
    if (cnt != kWalkCells && slots) {
        for_each_padded(C.nbr, C.n, t, cnt, C.cls_pos, [&](int q) { return fetch_at(C.cls_om, C.cls_nm, q); }, listed);
    } else if (cnt != kWalkCells) {
        for_each_padded(C.nbr, C.n, t, cnt, P, [&](int j) { return fetch_at(Om, Nm, j); }, listed);
    } else {
        walk_neighbors<Split>(
            i, pi, 0, P, grid_view(C, sc, off), C, Stage ? &S : nullptr, g,
            [&](int j, float4 pj4) { return j != i && phase_of(pj4) == phi && len2(pi - f3(pj4)) <= C.h2; },
            body);
    }
    finish_post_b(C, slots, i, t, vi4, eta, ft, Om, Vout);
}

template <bool Split, bool Stage, bool Persist = false>
__global__ void __launch_bounds__(kScanThreads, BP_POSTBC_MIN_BLOCKS) k_post_b(
    SimConsts C,
    const float4 *__restrict__ P,
    const float4 *__restrict__ V,
    const float4 *__restrict__ Om,
    const float4 *__restrict__ Nm,
    const int *__restrict__ off,
    float4 *__restrict__ Vout)
{
    // one tile of blockDim.x particles per CTA, or, persistent (an unstaged
    // launch of at most one resident wave: SimConsts::scan_persist), every
    // gridDim.x-th tile from blockIdx.x on
    if constexpr (Persist) {
        for (int i0 = blockIdx.x * blockDim.x; i0 < C.n; i0 += gridDim.x * blockDim.x)
            k_post_b_tile<Split, Stage>(C, P, V, Om, Nm, off, Vout, i0);
    } else {
        k_post_b_tile<Split, Stage>(C, P, V, Om, Nm, off, Vout, blockIdx.x * blockDim.x);
    }
}

// Pass C: XSPH viscosity (fluidXSph): same phase, j != i, r^2 <= h^2 (r = 0
// included).  Textbook mode weights each neighbour by its volume m_j / rho_j.
// First: no pass A or B before it, over the substep lists (k_post_c_lists).
template <bool Split, bool Stage, bool First = false>
__device__ __forceinline__ void k_post_c_tile(
    const SimConsts &C,
    const float4 *__restrict__ P,
    const float4 *__restrict__ V,
    const int *__restrict__ off,
    const float *__restrict__ mass,
    const float *__restrict__ rho,
    float4 *__restrict__ Vout,
    int i0)
{
    StageShared &S = stage_shared();
    const int t = i0 + threadIdx.x;
    const int i = (Stage || t >= C.n) ? t : walker_index(C, t);
    const float4 *__restrict__ vslots = First ? C.cls_vel : C.cls_vb;  // the velocities in class order
    int cnt = First ? 0 : post_list_count(C, P, i, t);
    const int g = (Stage && __syncthreads_or(cnt == kWalkCells)) ? stage_block(C, P, off, i0, S) : -1;
    if (i >= C.n) return;
    const float4 pi4 = P[i];
    const float4 vi4 = V[i];
    const int phi = phase_of(pi4);
    if (phi >= 0) {
        Vout[i] = vi4;
        return;
    }
    const float3 pi = f3(pi4), vi = f3(vi4);
    const GridView gv = grid_view(C, scene_index(C, i), off);
    if constexpr (First) {
        if (walk_mode(C)) {
            note_substep_list(C, t, i, pi, cell_of(pi, C), gv);
            cnt = kWalkCells;
        } else {
            if (!reads_substep_list(C, t, i, pi, cell_of(pi, C), gv)) return;
            cnt = __ldg(C.nbr_count + t) & 0xffff;
        }
    }
    float3 vn = make_float3(0.f, 0.f, 0.f);
    auto body_at = [&](const float4 *__restrict__ Vp, const float *__restrict__ mp, const float *__restrict__ rp,
                       int j, float4 pj4) {
        float wgt = poly6(C, len2(pi - f3(pj4)));
        if (C.textbook) wgt = __fmul_rn(wgt, __fdiv_rn(__ldg(mp + j), __ldg(rp + j)));
        vn = fma3(wgt, f3(Vp[j]) - vi, vn);
    };
    auto body = [&](int j, float4 pj4) { body_at(V, mass, rho, j, pj4); };
    auto test = [&](int j, float4 pj4) { return j != i && phase_of(pj4) == phi && len2(pi - f3(pj4)) <= C.h2; };
    int own = -1;
    // reference mode: each entry's velocity loads with its position, before
    // the four pair terms of a record
    // substep lists also hold the own entry, other phases and entries past h
    const int me = post_slots(C, Stage) ? t : i;
    auto keep = [&](int j, float4 pj4, float d2) { return j != me && phase_of(pj4) == phi && d2 <= C.h2; };
    auto listed = [&](int j, float4 pj4, float4 vj4) {
        const float d2 = len2(pi - f3(pj4));
        if (keep(j, pj4, d2)) vn = fma3(poly6(C, d2), f3(vj4) - vi, vn);
    };
    if (cnt != kWalkCells && post_slots(C, Stage) && !C.textbook) {  
        for_each_padded(C.nbr, C.n, t, cnt, C.cls_pos, [&](int q) { return vslots[q]; }, listed);
    } else if (cnt != kWalkCells && !C.textbook) {
        for_each_padded(C.nbr, C.n, t, cnt, P, [&](int j) { return V[j]; }, listed);
    } else if (cnt != kWalkCells && post_slots(C, Stage)) {
        for_each_in_list(C.nbr, C.n, t, cnt, C.cls_pos,
                         [&](int q, float4 pj4) {
                             if (keep(q, pj4, len2(pi - f3(pj4)))) body_at(vslots, C.cls_mass, C.cls_rho, q, pj4);
                         });
    } else if (cnt != kWalkCells) {
        for_each_in_list(C.nbr, C.n, t, cnt, P, [&](int j, float4 pj4) {
            if (keep(j, pj4, len2(pi - f3(pj4)))) body(j, pj4);
        });
    } else if (C.nbr && (First || !C.nbr_count)) {
        // no pass A before it: record the walk's pairs, then sum over them
        ListWriter list(C.nbr, C.nbr_cap, C.n, t);
        walk_neighbors<Split>(i, pi, 0, P, gv, C, Stage ? &S : nullptr, g, test, [&](int j, float4) { list.push(j); });
        own = list.finish();
        if (own >= 0) for_each_in_list<false>(C.nbr, C.n, t, own, P, body);
    }
    if (cnt == kWalkCells && own < 0) walk_neighbors<Split>(i, pi, 0, P, gv, C, Stage ? &S : nullptr, g, test, body);
    const float3 v = vi + C.xsph_c * vn;
    Vout[i] = make_float4(v.x, v.y, v.z, vi4.w);
}

template <bool Split, bool Stage, bool Persist = false>
__global__ void __launch_bounds__(kScanThreads, BP_POSTBC_MIN_BLOCKS) k_post_c(
    SimConsts C,
    const float4 *__restrict__ P,
    const float4 *__restrict__ V,
    const int *__restrict__ off,
    const float *__restrict__ mass,
    const float *__restrict__ rho,
    float4 *__restrict__ Vout)
{
    // one tile of blockDim.x particles per CTA, or, persistent (an unstaged
    // launch of at most one resident wave: SimConsts::scan_persist), every
    // gridDim.x-th tile from blockIdx.x on
    if constexpr (Persist) {
        for (int i0 = blockIdx.x * blockDim.x; i0 < C.n; i0 += gridDim.x * blockDim.x)
            k_post_c_tile<Split, Stage>(C, P, V, off, mass, rho, Vout, i0);
    } else {
        k_post_c_tile<Split, Stage>(C, P, V, off, mass, rho, Vout, blockIdx.x * blockDim.x);
    }
}

// A neighbour's velocity and density, as pass A's pair terms read them.
struct PostANeighbour {
    float3 v;
    float rho;
};
__device__ __forceinline__ PostANeighbour post_a_neighbour(const SimConsts &C, const float4 *__restrict__ V,
                                                           const float *__restrict__ rho, int j)
{
    PostANeighbour r;
    r.v = C.use_vort ? f3(V[j]) : make_float3(0.f, 0.f, 0.f);
    r.rho = C.use_akinci ? __ldg(rho + j) : 0.f;
    return r;
}
__device__ __forceinline__ void finish_post_a(const SimConsts &C, bool slots, int i, int t, float3 om, float3 nn,
                                              const float *__restrict__ rho, float4 *__restrict__ Om,
                                              float4 *__restrict__ Nm)
{
    const float4 om4 = make_float4(om.x, om.y, om.z, len3(om));
    const float3 n = C.h * nn;
    const float4 nm4 = make_float4(n.x, n.y, n.z, rho[i]);
    Om[i] = om4;
    Nm[i] = nm4;
    if (slots) {
        C.cls_om[t] = om4;
        C.cls_nm[t] = nm4;
    }
}

// Pass A over the substep lists: the sums of k_post_a, from the same pairs in
// the same order (post_slots() equals classes_on() with them).
__global__ void __launch_bounds__(kScanThreads, BP_POSTBC_MIN_BLOCKS) k_post_a_lists(
    SimConsts C, const float4 *__restrict__ P, const float4 *__restrict__ V, const float *__restrict__ rho,
    const int *__restrict__ off, float4 *__restrict__ Om, float4 *__restrict__ Nm)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= C.n) return;
    const bool slots = post_slots(C, false);
    const int i = slots ? __ldg(C.cls_perm + t) : t;
    const float4 pi4 = slots ? C.cls_pos[t] : P[i];
    const int phi = phase_of(pi4);
    if (phi >= 0) return;
    const float3 pi = f3(pi4);
    if (walk_mode(C)) {  // k_post_a_walks follows
        note_substep_list(C, t, i, pi, cell_of(pi, C), grid_view(C, scene_index(C, i), off));
        return;
    }
    if (!reads_substep_list(C, t, i, pi, cell_of(pi, C), grid_view(C, scene_index(C, i), off))) return;
    const int cnt = __ldg(C.nbr_count + t) & 0xffff;
    const float4 *__restrict__ src = slots ? C.cls_pos : P;
    const float4 *__restrict__ vs = slots ? C.cls_vel : V;
    const float *__restrict__ rs = slots ? C.cls_rho : rho;
    const float3 vi = f3(vs[t]);
    float3 om = make_float3(0.f, 0.f, 0.f), nn = make_float3(0.f, 0.f, 0.f);
    for_each_padded(
        C.nbr, C.n, t, cnt, src, [&](int j) { return post_a_neighbour(C, vs, rs, j); },
        [&](int, float4 pj4, const PostANeighbour &nb) {
            const float3 diff = pi - f3(pj4);
            const float d2 = len2(diff);
            const bool ok = d2 > 0.f && d2 <= C.h2 && phase_of(pj4) == phi;
            const float3 g = spiky_grad_r(C, diff, d2, rsqrtf(d2));
            const float3 w = cross3(nb.v - vi, g);
            if (ok && C.use_vort) om += w;
            if (ok && C.use_akinci) nn = fma3(__frcp_rn(nb.rho), g, nn);
        });
    finish_post_a(C, slots, i, t, om, nn, rho, Om, Nm);
}

// Pass A in walk mode, a launch of its own: k_post_a_lists' 3 CTAs an SM cost the
// walk 16 % (829,440 squeezed particles, 288 and 249 us), and where lists are
// read its early exit takes 2 us.
__global__ void __launch_bounds__(kScanThreads, BP_SCAN_MIN_BLOCKS) k_post_a_walks(
    SimConsts C, const float4 *__restrict__ P, const float4 *__restrict__ V, const float *__restrict__ rho,
    const int *__restrict__ off, float4 *__restrict__ Om, float4 *__restrict__ Nm)
{
    if (walk_mode(C)) k_post_a_tile<true, false>(C, P, V, rho, off, Om, Nm, blockIdx.x * blockDim.x);
}

// The queued particles' pass A, as k_lambda_queued: a queued particle leaves
// its neighbours within h in its list for passes B and C.
__global__ void __launch_bounds__(kQueueThreads) k_post_a_queued(SimConsts C, const float4 *__restrict__ P,
                                                                const float4 *__restrict__ V,
                                                                const float *__restrict__ rho,
                                                                const int *__restrict__ off, float4 *__restrict__ Om,
                                                                float4 *__restrict__ Nm)
{
    __shared__ WarpRows rows[kQueueThreads / 32];
    __shared__ WarpHits hits[kQueueThreads / 32];
    const int lane = threadIdx.x & 31;
    const int queued = C.sl_count[C.sl_pass];
    adapt_skin(C);
    const bool slots = post_slots(C, false);
    const float4 *__restrict__ vs = slots ? C.cls_vel : V;
    const float *__restrict__ rs = slots ? C.cls_rho : rho;
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) / 32; k < queued; k += gridDim.x * blockDim.x / 32) {
        const int t = C.sl_queue[k];
        const int i = slots ? __ldg(C.cls_perm + t) : t;
        const float4 pi4 = slots ? C.cls_pos[t] : P[i];
        const int phi = phase_of(pi4);
        const float3 pi = f3(pi4), vi = f3(vs[t]);
        if (C.nl_stats && slots && lane == 0) atomicAdd(C.nl_stats + 4, 1u);
        float acc = 0.f;  // lanes 0..2: omega, 3..5: the normal
        auto test = [&](int q, float4 pj) { return len2(pi - f3(pj)) <= C.h2 && phase_of(pj) == phi && q != t; };
        auto batch = [&](int k0, int n, int q, float4 pj) {
            const bool in = lane < n;
            if (in) put_entry(C, t, k0 + lane, q);
            float value[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            float scale = 0.f;
            const float3 diff = pi - f3(pj);
            const float d2 = len2(diff);
            const bool apart = in && d2 > 0.f;
            if (apart) {
                const PostANeighbour nb = post_a_neighbour(C, vs, rs, q);
                const float3 g = spiky_grad_r(C, diff, d2, rsqrtf(d2));
                const float3 w = cross3(nb.v - vi, g);
                value[0] = w.x;
                value[1] = w.y;
                value[2] = w.z;
                value[3] = g.x;
                value[4] = g.y;
                value[5] = g.z;
                scale = __frcp_rn(nb.rho);
            }
            warp_add<6, 3>(rows[threadIdx.x >> 5], __ballot_sync(kWarp, apart), value, scale, acc);
        };
        const int cnt = warp_neighbors(C, slots, cell_of(pi, C), P, grid_view(C, scene_index(C, i), off),
                                       hits[threadIdx.x >> 5], test, batch);
        warp_pad(C, t, cnt, t);
        float sum[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) sum[q] = __shfl_sync(kWarp, acc, q);
        if (lane != 0) continue;
        C.nbr_count[t] = cnt <= C.nbr_cap ? cnt : -1;
        const float3 zero = make_float3(0.f, 0.f, 0.f);
        finish_post_a(C, slots, i, t, C.use_vort ? make_float3(sum[0], sum[1], sum[2]) : zero,
                      C.use_akinci ? make_float3(sum[3], sum[4], sum[5]) : zero, rho, Om, Nm);
    }
}

// Pass C alone after the commit, over the substep lists: without pass A to ask
// which lists still hold, it asks itself, and its own queue follows.
// 65,536 particles, a launch: 46 us recording and summing its own walk, 15 us
// over the lists and 10 us for the queue.
__global__ void __launch_bounds__(kScanThreads, BP_POSTBC_MIN_BLOCKS) k_post_c_lists(
    SimConsts C, const float4 *__restrict__ P, const float4 *__restrict__ V, const int *__restrict__ off,
    const float *__restrict__ mass, const float *__restrict__ rho, float4 *__restrict__ Vout)
{
    k_post_c_tile<true, false, true>(C, P, V, off, mass, rho, Vout, blockIdx.x * blockDim.x);
}

__global__ void __launch_bounds__(kQueueThreads) k_post_c_queued(SimConsts C, const float4 *__restrict__ P,
                                                                const float4 *__restrict__ V,
                                                                const int *__restrict__ off,
                                                                const float *__restrict__ mass,
                                                                const float *__restrict__ rho,
                                                                float4 *__restrict__ Vout)
{
    __shared__ WarpRows rows[kQueueThreads / 32];
    __shared__ WarpHits hits[kQueueThreads / 32];
    const int lane = threadIdx.x & 31;
    const int queued = C.sl_count[C.sl_pass];
    adapt_skin(C);
    const bool slots = post_slots(C, false);
    const float4 *__restrict__ vs = slots ? C.cls_vel : V;
    const float *__restrict__ ms = slots ? C.cls_mass : mass;
    const float *__restrict__ rs = slots ? C.cls_rho : rho;
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) / 32; k < queued; k += gridDim.x * blockDim.x / 32) {
        const int t = C.sl_queue[k];
        const int i = slots ? __ldg(C.cls_perm + t) : t;
        const float4 pi4 = slots ? C.cls_pos[t] : P[i];
        const int phi = phase_of(pi4);
        const float4 vi4 = V[i];
        const float3 pi = f3(pi4), vi = f3(vi4);
        if (C.nl_stats && slots && lane == 0) atomicAdd(C.nl_stats + 4, 1u);
        float acc = 0.f;  // lanes 0..2: the weighted velocity differences
        auto test = [&](int q, float4 pj) { return q != t && phase_of(pj) == phi && len2(pi - f3(pj)) <= C.h2; };
        auto batch = [&](int, int n, int q, float4 pj) {
            const bool in = lane < n;
            float value[3] = {0.f, 0.f, 0.f};
            float wgt = 0.f;
            if (in) {
                wgt = poly6(C, len2(pi - f3(pj)));
                if (C.textbook) wgt = __fmul_rn(wgt, __fdiv_rn(__ldg(ms + q), __ldg(rs + q)));
                const float3 dv = f3(vs[q]) - vi;
                value[0] = dv.x;
                value[1] = dv.y;
                value[2] = dv.z;
            }
            warp_add<3, 0>(rows[threadIdx.x >> 5], __ballot_sync(kWarp, in), value, wgt, acc);
        };
        warp_neighbors(C, slots, cell_of(pi, C), P, grid_view(C, scene_index(C, i), off), hits[threadIdx.x >> 5], test,
                       batch);
        const float3 vn = make_float3(__shfl_sync(kWarp, acc, 0), __shfl_sync(kWarp, acc, 1), __shfl_sync(kWarp, acc, 2));
        if (lane != 0) continue;
        const float3 v = vi + C.xsph_c * vn;
        Vout[i] = make_float4(v.x, v.y, v.z, vi4.w);
    }
}

// The recording pass of small scenes, a warp per particle (k_lambda_lists<
// kRecordLists> takes a thread's whole walk, about 28 us whatever the number of
// particles): the candidates within the lists' reach, from the position
// records, the contact partners among them and, for fluid, the lambda pass's
// sums over those within h.
// Measured, a frame (a thread each, a warp each): 1,728 particles 188 -> 157
// us, 5,832 200 -> 177, 13,824 232 -> 233 (textbook mode 327 -> 315), 21,952
// 276 -> 296: the line lies at kWarpRecordMax.
constexpr int kWarpRecordMax = 14000;
__global__ void __launch_bounds__(kQueueThreads) k_lambda_record(SimConsts C, const float4 *__restrict__ P,
                                                                 const float *__restrict__ mass,
                                                                 const int *__restrict__ off, float *__restrict__ lam,
                                                                 float *__restrict__ rho)
{
    __shared__ WarpRows rows[kQueueThreads / 32];
    __shared__ WarpHits hits[kQueueThreads / 32];
    const int lane = threadIdx.x & 31;
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        C.sl_count[0] = C.sl_count[1] = C.sl_count[kSlDisplaced] = C.sl_count[kSlWalks] = C.sl_count[kSlContactWalks] = 0;
        C.sl_count[kSlMoved] = C.cls_perm ? *C.cls_moved : 0;
    }
    if (t >= C.n) return;  // whole warps
    const bool slots = classes_on(C);
    const int i = slots ? __ldg(C.cls_perm + t) : t;
    const float4 pi4 = slots ? C.cls_pos[t] : P[i];
    const float3 pi = f3(pi4);
    const int phi = phase_of(pi4);
    const bool solid = phi > 0;
    if (lane == 0) {
        C.sl_pos[i] = pi4;
        if (solid && C.sl_fluid) record_solid(C, slots, i, t, mass, lam);
    }
    if (solid && C.textbook && !C.cl_list) return;  // as lambda_substep_list
    const int sc = scene_index(C, i);
    const GridView v = grid_view(C, sc, off);
    const int3 c = cell_of(pi, C);
    if (C.nl_stats && lane == 0) {
        atomicAdd(C.nl_stats + 1, 1u);
        if (slots) atomicAdd(C.nl_stats + 4, 1u);
    }
    const float skin = substep_skin(C), touch = 2.0f * C.radius + skin;
    const float reach = fmaxf(C.sl_fluid ? C.h + skin : 0.f, C.cl_list ? touch : 0.f);
    const float reach2 = __fmul_rn(reach, reach), touch2 = __fmul_rn(touch, touch);
    const float inv_rho0 = inv_rest_density(C, sc);
    const int me = slots ? t : i;
    const bool sums = C.sl_fluid && !solid;
    float acc = 0.f;  // lane 0: the density; textbook, lanes 1..4: sum of g^2, -sum of g
    int self = kNoOwnEntry, touching = 0;
    auto batch = [&](int k0, int n, int q, float4 pj) {
        const bool in = lane < n;
        if (in) put_entry(C, t, k0 + lane, q);
        const unsigned own = __ballot_sync(kWarp, in && q == me);
        if (own) self = k0 + __ffs(own) - 1;
        const float3 diff = pi - f3(pj);
        const float d2 = len2(diff);
        if (C.cl_list) {
            const int phj = phase_of(pj);
            const bool near = in && phi != phj && (solid || phj > 0) && d2 <= touch2;
            const unsigned b = __ballot_sync(kWarp, near);
            const int k = touching + __popc(b & ((1u << lane) - 1u));
            if (near && k < kContactCap) C.cl_list[(size_t)k * C.n + t] = slots ? __ldg(C.cls_perm + q) : q;
            touching += __popc(b);
        }
        if (!sums) return;
        bool take = in && d2 <= C.h2;
        float value[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
        if (take) {
            const int j = slots ? __ldg(C.cls_perm + q) : q;
            const float mj = __ldg((slots ? C.cls_mass : mass) + q);
            take = C.textbook || j >= i;
            value[0] = __fmul_rn(mj, poly6(C, d2));
            if (phase_of(pj) >= 0) value[0] = __fmul_rn(C.solid_scale, value[0]);
            if (C.textbook && d2 > 0.f) {  // the pair at r = 0 adds zeros
                const float3 g = __fmul_rn(-mj, inv_rho0) * spiky_grad_r(C, diff, d2, rsqrtf(d2));
                value[1] = dot3(g, g);
                value[2] = -g.x;
                value[3] = -g.y;
                value[4] = -g.z;
            }
        }
        warp_add(rows[threadIdx.x >> 5], __ballot_sync(kWarp, take), value, 1.f, acc);
    };
    int cnt = warp_neighbors(C, slots, c, P, v, hits[threadIdx.x >> 5],
                             [&](int, float4 pj) { return len2(pi - f3(pj)) <= reach2; }, batch);
    const bool fits = cnt <= C.nbr_cap;
    if (!fits && C.sl_fluid)  // the neighbours within h alone may still fit; later passes then walk
        cnt = warp_neighbors(C, slots, c, P, v, hits[threadIdx.x >> 5],
                             [&](int, float4 pj) { return len2(pi - f3(pj)) <= C.h2; },
                             [&](int k0, int n, int q, float4) {
                                 if (lane < n) put_entry(C, t, k0 + lane, q);
                                 const unsigned own = __ballot_sync(kWarp, lane < n && q == me);
                                 if (own) self = k0 + __ffs(own) - 1;
                             });
    warp_pad(C, t, cnt, me);
    const float sum_g2 = __shfl_sync(kWarp, acc, 1);
    const float3 gi = make_float3(__shfl_sync(kWarp, acc, 2), __shfl_sync(kWarp, acc, 3), __shfl_sync(kWarp, acc, 4));
    if (lane != 0) return;
    C.nbr_count[t] = cnt <= C.nbr_cap ? cnt | (self << 16) : -1;
    C.sl_cell[t] = (fits && near_stored_cell(C, i, c, v)) ? v.base + cell_addr(c.x, c.y, c.z, v.D, v.mask) : kListNone;
    if (C.cl_list) C.cl_count[t] = fits && touching <= kContactCap ? touching : -1;
    if (sums)
        finish_lambda(C, slots, i, t, acc, rest_density(C, sc),
                      C.textbook ? (sum_g2 + dot3(gi, gi)) + C.relaxation : C.lambda_den, mass, lam, rho);
}

// ---- the list readers of small scenes: four lanes per particle ----

// A reading pass's thread takes its list's records one after another, a round
// of gathers and four pair terms each, and in a scene whose particles do not
// fill the GPU nothing hides that chain.  Four lanes per particle take four
// records at once and add their terms up in turn, in list order and with the
// same operations, so to the same bits (fma(1, v, s) rounds as v + s).
// Measured, a frame (one thread each, four lanes): 1,728 particles 244 -> 184
// us, 21,952 particles 307 -> 275, 32,768 301 -> 306; textbook mode, whose
// lambda pass has more to add up, 421 -> 274, 505 -> 387, 510 -> 448 and 46,656
// particles 567 -> 566: the lines lie just below.
constexpr int kGroupLanes = 4, kGroupThreads = 128;
constexpr int kGroupMax = 30000, kGroupMaxTextbook = 45000;

// A pair's addends: component k adds s[k / 3] * v[k].
template <int NV>
struct GroupTerm {
    float v[NV];
    float s[2];
};
struct GroupParticle {
    int t, i, lane;  // slot, sorted index, lane in the group
    bool slots, real;
    float4 p4;
};
// Lanes past the end repeat the last particle and store nothing (real).
__device__ __forceinline__ GroupParticle group_particle(const SimConsts &C, const float4 *__restrict__ P, bool slots)
{
    GroupParticle g;
    const int t = (blockIdx.x * kGroupThreads + threadIdx.x) / kGroupLanes;
    g.lane = threadIdx.x % kGroupLanes;
    g.real = t < C.n;
    g.t = min(t, C.n - 1);
    g.slots = slots;
    g.i = slots ? __ldg(C.cls_perm + g.t) : g.t;
    g.p4 = slots ? C.cls_pos[g.t] : P[g.i];
    return g;
}

// acc += the terms of entries [4 * first, cnt) of the particle's list, in
// order, on every lane: term(j, e, P[j], fetch(j), out) is false where entry e
// adds nothing.  All lanes of the warp take part (cnt 0: none to add).
template <int NV, class G, class F>
__device__ __forceinline__ void group_sum(const SimConsts &C, const GroupParticle &me, int first, int cnt,
                                          const float4 *__restrict__ P, G &&fetch, F &&term, float (&acc)[NV])
{
    using X = decltype(fetch(0));
    const int recs = (cnt + 3) >> 2;
    const int4 *rec = reinterpret_cast<const int4 *>(C.nbr) + me.t;
    const size_t stride = (size_t)C.n;
    const int own = me.slots ? me.t : me.i;
    const int rounds = __reduce_max_sync(kWarp, max(recs - first + kGroupLanes - 1, 0) / kGroupLanes);
    int at = first + me.lane;
    int4 next = at < recs ? __ldg(rec + (size_t)at * stride) : make_int4(own, own, own, own);
    for (int r = 0; r < rounds; ++r, at += kGroupLanes) {
        const int j[4] = {next.x, next.y, next.z, next.w};
        next = at + kGroupLanes < recs ? __ldg(rec + (size_t)(at + kGroupLanes) * stride) : make_int4(own, own, own, own);
        float4 pj[4];
        X xj[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            pj[q] = P[j[q]];
            xj[q] = fetch(j[q]);
        }
        GroupTerm<NV> g[4];
        bool ok[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) ok[q] = term(j[q], 4 * at + q, pj[q], xj[q], g[q]) && at < recs;
#pragma unroll
        for (int l = 0; l < kGroupLanes; ++l) {
            if (me.lane == l) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (ok[q]) {
#pragma unroll
                        for (int k = 0; k < NV; ++k) acc[k] = __fmaf_rn(g[q].s[k / 3], g[q].v[k], acc[k]);
                    }
            }
#pragma unroll
            for (int k = 0; k < NV; ++k) acc[k] = __shfl_sync(kWarp, acc[k], l, kGroupLanes);
        }
    }
}

// One lane of the group asks whether the particle reads its list (and queues it where not).
__device__ __forceinline__ bool group_reads(const SimConsts &C, const GroupParticle &me, bool wanted, int3 c,
                                            const GridView &v)
{
    bool reads = false;
    if (me.lane == 0 && me.real && wanted) reads = reads_substep_list(C, me.t, me.i, f3(me.p4), c, v);
    return __shfl_sync(kWarp, reads, 0, kGroupLanes);
}

template <bool Textbook>
__global__ void __launch_bounds__(kGroupThreads) k_lambda_group(SimConsts C, const float4 *__restrict__ P,
                                                                const float *__restrict__ mass,
                                                                const int *__restrict__ off, float *__restrict__ lam,
                                                                float *__restrict__ rho)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) C.sl_count[C.sl_pass ^ 1] = 0;  // the next pass's queue
    const GroupParticle me = group_particle(C, P, classes_on(C));
    const bool solid = phase_of(me.p4) > 0;
    const float3 pi = f3(me.p4);
    const int sc = scene_index(C, me.i);
    const GridView v = grid_view(C, sc, off);
    const int3 c = cell_of(pi, C);
    const bool reads = group_reads(C, me, !(solid && Textbook), c, v) && !solid;
    const int packed = reads ? __ldg(C.nbr_count + me.t) : 0;
    const int cnt = packed & 0xffff, self = packed >> 16;
    const float *__restrict__ ms = me.slots ? C.cls_mass : mass;
    const float4 *__restrict__ src = me.slots ? C.cls_pos : P;
    auto fetch = [&](int j) { return __ldg(ms + j); };
    auto weight = [&](float mj, float4 pj, float d2) {
        const float ld = __fmul_rn(mj, poly6(C, d2));
        return (phase_of(pj) < 0) ? ld : __fmul_rn(C.solid_scale, ld);
    };
    float density, den = C.lambda_den;
    if (!Textbook) {
        auto inner = [&](int a) {
            const unsigned u = (unsigned)a & v.mask;
            return u != 0u && u != v.mask;
        };
        // as lambda_substep_list
        const bool ascending = self != kNoOwnEntry && inner(c.x) && inner(c.y) && inner(c.z);
        float acc[1] = {0.f};
        group_sum<1>(C, me, ascending ? self >> 2 : 0, cnt, src, fetch,
                     [&](int j, int e, float4 pj, float mj, GroupTerm<1> &out) {
            const float d2 = len2(pi - f3(pj));
            out.s[0] = 1.f;
            out.v[0] = weight(mj, pj, d2);
            if (!(d2 <= C.h2) || e >= cnt) return false;
            return ascending ? e >= self : (me.slots ? __ldg(C.cls_perm + j) : j) >= me.i;
        }, acc);
        density = acc[0];
    } else {
        const float inv_rho0 = inv_rest_density(C, sc);
        float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
        group_sum<5>(C, me, 0, cnt, src, fetch, [&](int, int e, float4 pj, float mj, GroupTerm<5> &out) {
            const float3 diff = pi - f3(pj);
            const float d2 = len2(diff);
            out.s[0] = out.s[1] = 1.f;
            out.v[0] = weight(mj, pj, d2);
            out.v[1] = out.v[2] = out.v[3] = out.v[4] = 0.f;  // r = 0 adds zeros
            if (d2 > 0.f) {
                const float3 g = __fmul_rn(-mj, inv_rho0) * spiky_grad_r(C, diff, d2, rsqrtf(d2));
                out.v[1] = dot3(g, g);
                out.v[2] = -g.x;
                out.v[3] = -g.y;
                out.v[4] = -g.z;
            }
            return d2 <= C.h2 && e < cnt;
        }, acc);
        density = acc[0];
        const float3 gi = make_float3(acc[2], acc[3], acc[4]);
        den = (acc[1] + dot3(gi, gi)) + C.relaxation;
    }
    if (reads && me.lane == 0) finish_lambda(C, me.slots, me.i, me.t, density, rest_density(C, sc), den, mass, lam, rho);
}

__global__ void __launch_bounds__(kGroupThreads) k_deltap_group(SimConsts C, DeltaArgs a)
{
    const GroupParticle me = group_particle(C, a.P, classes_on(C));
    const int phk = phase_of(me.p4);
    const float3 pk = f3(me.p4);
    const bool moves = !(C.textbook && phk > 0);
    const int listed = moves ? __ldg(C.nbr_count + me.t) : 0;
    const float lk = a.lam[me.i];
    const float2 *__restrict__ lms = me.slots ? C.cls_lm : C.lm;
    float3 sum;
    auto pair = [&](float3 diff, float d2, float lj) {
        float sl = __fadd_rn(lk, lj);
        if (C.scorr_on)
            sl = __fsub_rn(sl, __fmul_rn(C.scorr_k, ipowf(__fmul_rn(poly6(C, d2), C.scorr_inv_wq), C.scorr_ni)));
        float3 delta = sl * spiky_grad_r(C, diff, d2, rsqrtf(d2));
        if (C.delta_clamp > 0.f) {
            const float l2 = len2(delta);
            if (!(l2 < C.delta_clamp2)) delta = delta * __fmul_rn(C.delta_clamp, rsqrtf(l2));
        }
        return delta;
    };
    // reference mode: the lower-indexed of the pair is fluid
    auto admits = [&](int j, bool fj) { return C.textbook || ((j > me.i) ? (phk < 0) : fj); };
    float acc[3] = {0.f, 0.f, 0.f};
    group_sum<3>(C, me, 0, listed >= 0 ? listed & 0xffff : 0, me.slots ? C.cls_pos : a.P,
                 [&](int j) { return __ldg(lms + j); },
                 [&](int j, int, float4 pj, float2 lm, GroupTerm<3> &out) {
        const float3 diff = pk - f3(pj);
        const float d2 = len2(diff);
        const float3 delta = pair(diff, d2, lm.x);
        out.s[0] = lm.y;
        out.v[0] = delta.x;
        out.v[1] = delta.y;
        out.v[2] = delta.z;
        const bool fj = phase_of(pj) < 0;
        return d2 > 0.f && d2 <= C.h2 && ((phk < 0 && fj) || admits(me.slots ? __ldg(C.cls_perm + j) : j, fj));
    }, acc);
    if (me.lane != 0 || !me.real) return;
    sum = make_float3(acc[0], acc[1], acc[2]);
    const int sc = scene_index(C, me.i);
    if (listed < 0)  // overflowed
        walk_neighbors<true>(
            me.i, pk, 0, a.P, grid_view(C, sc, a.off), C, nullptr, -1,
            [&](int, float4 pj) {
                const float d2 = len2(pk - f3(pj));
                return d2 <= C.h2 && d2 > 0.f;
            },
            [&](int j, float4 pj) {
                if (!admits(j, phase_of(pj) < 0)) return;
                const float3 diff = pk - f3(pj);
                sum = fma3(__ldg(a.mass + j), pair(diff, len2(diff), __ldg(a.lam + j)), sum);
            });
    finish_deltap(C, a, sc, me.i, me.p4, sum);
}

__global__ void __launch_bounds__(kGroupThreads) k_post_a_group(SimConsts C, const float4 *__restrict__ P,
                                                                const float4 *__restrict__ V,
                                                                const float *__restrict__ rho,
                                                                const int *__restrict__ off, float4 *__restrict__ Om,
                                                                float4 *__restrict__ Nm)
{
    const GroupParticle me = group_particle(C, P, post_slots(C, false));
    const int phi = phase_of(me.p4);
    const float3 pi = f3(me.p4);
    const bool reads = group_reads(C, me, phi < 0, cell_of(pi, C), grid_view(C, scene_index(C, me.i), off));
    const int cnt = reads ? __ldg(C.nbr_count + me.t) & 0xffff : 0;
    const float4 *__restrict__ vs = me.slots ? C.cls_vel : V;
    const float *__restrict__ rs = me.slots ? C.cls_rho : rho;
    const float3 vi = f3(vs[me.t]);
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    group_sum<6>(C, me, 0, cnt, me.slots ? C.cls_pos : P, [&](int j) { return post_a_neighbour(C, vs, rs, j); },
                 [&](int, int, float4 pj, const PostANeighbour &nb, GroupTerm<6> &out) {
        const float3 diff = pi - f3(pj);
        const float d2 = len2(diff);
        const float3 g = spiky_grad_r(C, diff, d2, rsqrtf(d2));
        const float3 w = cross3(nb.v - vi, g);
        out.s[0] = 1.f;
        out.s[1] = __frcp_rn(nb.rho);
        out.v[0] = w.x;
        out.v[1] = w.y;
        out.v[2] = w.z;
        out.v[3] = g.x;
        out.v[4] = g.y;
        out.v[5] = g.z;
        return d2 > 0.f && d2 <= C.h2 && phase_of(pj) == phi;
    }, acc);
    if (!reads || me.lane != 0) return;
    const float3 zero = make_float3(0.f, 0.f, 0.f);
    finish_post_a(C, me.slots, me.i, me.t, C.use_vort ? make_float3(acc[0], acc[1], acc[2]) : zero,
                  C.use_akinci ? make_float3(acc[3], acc[4], acc[5]) : zero, rho, Om, Nm);
}

__global__ void __launch_bounds__(kGroupThreads) k_post_b_group(SimConsts C, const float4 *__restrict__ P,
                                                                const float4 *__restrict__ V,
                                                                const float4 *__restrict__ Om,
                                                                const float4 *__restrict__ Nm,
                                                                const int *__restrict__ off, float4 *__restrict__ Vout)
{
    const GroupParticle me = group_particle(C, P, post_slots(C, false));
    const int phi = phase_of(me.p4);
    const float3 pi = f3(me.p4);
    const float4 vi4 = V[me.i];
    const float4 ni4 = Nm[me.i];
    const int sc = scene_index(C, me.i);
    const float two_rho0 = 2.0f * rest_density(C, sc);
    const int listed = phi < 0 ? __ldg(C.nbr_count + me.t) : 0;
    const bool want_v = C.use_vort, want_t = C.use_akinci;
    struct Nb {
        float om;
        float4 nm;
    };
    auto fetch_at = [&](const float4 *__restrict__ Omp, const float4 *__restrict__ Nmp, int j) {
        Nb r;
        r.om = want_v ? Omp[j].w : 0.f;
        r.nm = want_t ? Nmp[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        return r;
    };
    auto term = [&](float4 pj, const Nb &nb, GroupTerm<6> &out) {
        const float3 diff = pi - f3(pj);
        const float d2 = len2(diff);
        const float inv_r = rsqrtf(d2);
        const float3 g = spiky_grad_r(C, diff, d2, inv_r);
        const float dist = __fmul_rn(d2, inv_r);
        const float3 fco = __fmul_rn(__fmul_rn(-C.tension, akinci_spline(C, dist)), inv_r) * diff;
        const float3 f = fco + (-C.tension) * (f3(ni4) - f3(nb.nm));
        out.s[0] = nb.om;
        out.s[1] = __fmul_rn(two_rho0, __frcp_rn(__fadd_rn(ni4.w, nb.nm.w)));
        out.v[0] = g.x;
        out.v[1] = g.y;
        out.v[2] = g.z;
        out.v[3] = f.x;
        out.v[4] = f.y;
        out.v[5] = f.z;
        return d2 > 0.f && d2 <= C.h2 && phase_of(pj) == phi;
    };
    const float4 *__restrict__ oms = me.slots ? C.cls_om : Om;
    const float4 *__restrict__ nms = me.slots ? C.cls_nm : Nm;
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    group_sum<6>(C, me, 0, listed >= 0 ? listed & 0xffff : 0, me.slots ? C.cls_pos : P,
                 [&](int j) { return fetch_at(oms, nms, j); },
                 [&](int, int, float4 pj, const Nb &nb, GroupTerm<6> &out) { return term(pj, nb, out); }, acc);
    if (me.lane != 0 || !me.real) return;
    if (phi >= 0) {
        Vout[me.i] = vi4;
        return;
    }
    if (listed < 0)  // overflowed
        walk_neighbors<true>(
            me.i, pi, 0, P, grid_view(C, sc, off), C, nullptr, -1,
            [&](int j, float4 pj) { return j != me.i && phase_of(pj) == phi && len2(pi - f3(pj)) <= C.h2; },
            [&](int j, float4 pj) {
                GroupTerm<6> out;
                if (!term(pj, fetch_at(Om, Nm, j), out)) return;
#pragma unroll
                for (int k = 0; k < 6; ++k) acc[k] = __fmaf_rn(out.s[k / 3], out.v[k], acc[k]);
            });
    finish_post_b(C, me.slots, me.i, me.t, vi4, make_float3(acc[0], acc[1], acc[2]),
                  make_float3(acc[3], acc[4], acc[5]), Om, Vout);
}

template <bool First>  // as k_post_c_tile
__global__ void __launch_bounds__(kGroupThreads) k_post_c_group(SimConsts C, const float4 *__restrict__ P,
                                                                const float4 *__restrict__ V,
                                                                const int *__restrict__ off,
                                                                const float *__restrict__ mass,
                                                                const float *__restrict__ rho,
                                                                float4 *__restrict__ Vout)
{
    const GroupParticle me = group_particle(C, P, post_slots(C, false));
    const int phi = phase_of(me.p4);
    const float3 pi = f3(me.p4);
    const float4 vi4 = V[me.i];
    const float3 vi = f3(vi4);
    const GridView gv = grid_view(C, scene_index(C, me.i), off);
    const bool reads = First ? group_reads(C, me, phi < 0, cell_of(pi, C), gv) : phi < 0;
    const int listed = reads ? __ldg(C.nbr_count + me.t) : 0;
    const int own = me.slots ? me.t : me.i;
    struct Nb {
        float3 v;
        float m, rho;
    };
    auto fetch_at = [&](const float4 *__restrict__ Vp, const float *__restrict__ mp, const float *__restrict__ rp, int j) {
        Nb r;
        r.v = f3(Vp[j]);
        r.m = C.textbook ? __ldg(mp + j) : 0.f;
        r.rho = C.textbook ? __ldg(rp + j) : 1.f;
        return r;
    };
    auto term = [&](float4 pj, const Nb &nb, GroupTerm<3> &out) {
        const float d2 = len2(pi - f3(pj));
        float wgt = poly6(C, d2);
        if (C.textbook) wgt = __fmul_rn(wgt, __fdiv_rn(nb.m, nb.rho));
        const float3 dv = nb.v - vi;
        out.s[0] = wgt;
        out.v[0] = dv.x;
        out.v[1] = dv.y;
        out.v[2] = dv.z;
        return phase_of(pj) == phi && d2 <= C.h2;
    };
    const float4 *__restrict__ vs = me.slots ? (First ? C.cls_vel : C.cls_vb) : V;
    const float *__restrict__ ms = me.slots ? C.cls_mass : mass;
    const float *__restrict__ rs = me.slots ? C.cls_rho : rho;
    float acc[3] = {0.f, 0.f, 0.f};
    group_sum<3>(C, me, 0, listed >= 0 ? listed & 0xffff : 0, me.slots ? C.cls_pos : P,
                 [&](int j) { return fetch_at(vs, ms, rs, j); },
                 [&](int j, int, float4 pj, const Nb &nb, GroupTerm<3> &out) { return term(pj, nb, out) && j != own; }, acc);
    if (me.lane != 0 || !me.real) return;
    if (phi >= 0) {
        Vout[me.i] = vi4;
        return;
    }
    if (First && !reads) return;  // queued
    if (listed < 0)  // overflowed
        walk_neighbors<true>(
            me.i, pi, 0, P, gv, C, nullptr, -1,
            [&](int j, float4 pj) { return j != me.i && phase_of(pj) == phi && len2(pi - f3(pj)) <= C.h2; },
            [&](int j, float4 pj) {
                GroupTerm<3> out;
                if (!term(pj, fetch_at(V, mass, rho, j), out)) return;
#pragma unroll
                for (int k = 0; k < 3; ++k) acc[k] = __fmaf_rn(out.s[0], out.v[k], acc[k]);
            });
    const float3 v = vi + C.xsph_c * make_float3(acc[0], acc[1], acc[2]);
    Vout[me.i] = make_float4(v.x, v.y, v.z, vi4.w);
}

bool reads_in_groups(int n, bool textbook) { return n <= (textbook ? kGroupMaxTextbook : kGroupMax); }
static bool use_groups(const SimConsts &C) { return C.sl_pos && reads_in_groups(C.n, C.textbook != 0); }
static unsigned group_blocks(const SimConsts &C)
{
    return (unsigned)(((long long)C.n * kGroupLanes + kGroupThreads - 1) / kGroupThreads);
}

bool records_from_planes(int n) { return n > kWarpRecordMax; }

void launch_lambda_lists(cudaStream_t st, const SimConsts &C, bool record, const float4 *P, const float *mass,
                         const int *off, float *lam, float *rho, LaunchLog *L)
{
    if (C.n <= 0) return;
    const int grid = (C.n + C.scan_block - 1) / C.scan_block;
    if (record && C.n <= kWarpRecordMax) {
        k_lambda_record<<<(C.n * 32 + kQueueThreads - 1) / kQueueThreads, kQueueThreads, 0, st>>>(C, P, mass, off, lam,
                                                                                               rho);
        L->done("launch_lambda");
        return;
    }
    const bool walks = C.sl_may_walk != 0;
    if (record) {
        if (walks) k_lambda_lists<kRecordLists, true><<<grid, C.scan_block, 0, st>>>(C, P, mass, off, lam, rho);
        else k_lambda_lists<kRecordLists, false><<<grid, C.scan_block, 0, st>>>(C, P, mass, off, lam, rho);
        L->done("launch_lambda");
        return;
    }
    if (use_groups(C) && C.textbook)
        k_lambda_group<true><<<group_blocks(C), kGroupThreads, 0, st>>>(C, P, mass, off, lam, rho);
    else if (use_groups(C))
        k_lambda_group<false><<<group_blocks(C), kGroupThreads, 0, st>>>(C, P, mass, off, lam, rho);
    else if (walks) k_lambda_lists<kReadLists, true><<<grid, C.scan_block, 0, st>>>(C, P, mass, off, lam, rho);
    else k_lambda_lists<kReadLists, false><<<grid, C.scan_block, 0, st>>>(C, P, mass, off, lam, rho);
    L->done("launch_lambda_lists");
    k_lambda_queued<<<queue_blocks(C.n, kQueueThreads), kQueueThreads, 0, st>>>(C, P, mass, off, lam, rho);
    L->done("launch_lambda_queued");
}
void launch_deltap(cudaStream_t st, const SimConsts &C, const DeltaArgs &a, LaunchLog *L)
{
    if (C.n <= 0) return;
    if (use_groups(C)) k_deltap_group<<<group_blocks(C), kGroupThreads, 0, st>>>(C, a);
    else BP_LAUNCH_SPLIT(k_deltap, st, C, a);
    L->done(__func__);
}
void launch_post_a_lists(cudaStream_t st, const SimConsts &C, const float4 *P, const float4 *V, const float *rho,
                         const int *off, float4 *Om, float4 *Nm, LaunchLog *L)
{
    if (C.n <= 0) return;
    if (use_groups(C)) k_post_a_group<<<group_blocks(C), kGroupThreads, 0, st>>>(C, P, V, rho, off, Om, Nm);
    else k_post_a_lists<<<(C.n + C.scan_block - 1) / C.scan_block, C.scan_block, 0, st>>>(C, P, V, rho, off, Om, Nm);
    L->done("launch_post_a_lists");
    if (C.sl_may_walk) {
        k_post_a_walks<<<(C.n + C.scan_block - 1) / C.scan_block, C.scan_block, 0, st>>>(C, P, V, rho, off, Om, Nm);
        L->done("launch_post_a_walks");
    }
    k_post_a_queued<<<queue_blocks(C.n, kQueueThreads), kQueueThreads, 0, st>>>(C, P, V, rho, off, Om, Nm);
    L->done("launch_post_a_queued");
}
void launch_post_a(cudaStream_t st, const SimConsts &C, const float4 *P, const float4 *V, const float *rho,
                   const int *off, float4 *Om, float4 *Nm, LaunchLog *L)
{
    if (C.n <= 0) return;
    BP_LAUNCH_SPLIT(k_post_a, st, C, P, V, rho, off, Om, Nm);
    L->done(__func__);
}
void launch_post_b(cudaStream_t st, const SimConsts &C, const float4 *P, const float4 *V, const float4 *Om,
                   const float4 *Nm, const int *off, float4 *Vout, LaunchLog *L)
{
    if (C.n <= 0) return;
    if (use_groups(C)) k_post_b_group<<<group_blocks(C), kGroupThreads, 0, st>>>(C, P, V, Om, Nm, off, Vout);
    else BP_LAUNCH_SPLIT(k_post_b, st, C, P, V, Om, Nm, off, Vout);
    L->done(__func__);
}
void launch_post_c_lists(cudaStream_t st, const SimConsts &C, const float4 *P, const float4 *V, const int *off,
                         const float *mass, const float *rho, float4 *Vout, LaunchLog *L)
{
    if (C.n <= 0) return;
    if (use_groups(C)) k_post_c_group<true><<<group_blocks(C), kGroupThreads, 0, st>>>(C, P, V, off, mass, rho, Vout);
    else k_post_c_lists<<<(C.n + C.scan_block - 1) / C.scan_block, C.scan_block, 0, st>>>(C, P, V, off, mass, rho, Vout);
    L->done("launch_post_c_lists");
    k_post_c_queued<<<queue_blocks(C.n, kQueueThreads), kQueueThreads, 0, st>>>(C, P, V, off, mass, rho, Vout);
    L->done("launch_post_c_queued");
}
void launch_post_c(cudaStream_t st, const SimConsts &C, const float4 *P, const float4 *V, const int *off,
                   const float *mass, const float *rho, float4 *Vout, LaunchLog *L)
{
    if (C.n <= 0) return;
    if (use_groups(C) && C.nbr_count) k_post_c_group<false><<<group_blocks(C), kGroupThreads, 0, st>>>(C, P, V, off, mass, rho, Vout);
    else BP_LAUNCH_SPLIT(k_post_c, st, C, P, V, off, mass, rho, Vout);
    L->done(__func__);
}

// Same count on caller buffers in the reference's start/end format.  The three
// cells of a column are one run of sorted positions (their keys are
// consecutive), from the first occupied one's start to the last one's end: two
// loads find it where both ends are occupied, and its positions are read in
// order, Ahead of them (3 floats each) at a time.  Where the column wraps
// around the table, two of its cells are a run and the third follows alone.
// Bound by the latency and number of those loads (1,000,003 points, 128^3
// table: 92 us; cell by cell, 27 pairs of loads a point, 153 us; three 16-byte
// loads for four positions from the boundary below the run, 97 us).
template <int Ahead>
__device__ __forceinline__ int count_run(int b, int e, const float *__restrict__ pos3, float3 pi, float h2)
{
    int cnt = 0;
    for (; b + Ahead <= e; b += Ahead) {
        float v[3 * Ahead];
#pragma unroll
        for (int k = 0; k < 3 * Ahead; ++k) v[k] = __ldg(pos3 + 3 * (size_t)b + k);
#pragma unroll
        for (int k = 0; k < Ahead; ++k)
            cnt += len2(pi - make_float3(v[3 * k], v[3 * k + 1], v[3 * k + 2])) <= h2 ? 1 : 0;
    }
    if constexpr (Ahead > 4) return cnt + count_run<4>(b, e, pos3, pi, h2);
    for (; b < e; ++b) {
        const float *p = pos3 + 3 * (size_t)b;
        cnt += len2(pi - make_float3(__ldg(p), __ldg(p + 1), __ldg(p + 2))) <= h2 ? 1 : 0;
    }
    return cnt;
}

// The `cells` consecutive cells from a on (2 or 3).
template <int Ahead>
__device__ __forceinline__ int count_cells(int a, int cells, const int *__restrict__ start,
                                           const int *__restrict__ end, const float *__restrict__ pos3, float3 pi,
                                           float h2)
{
    const int last = a + cells - 1;
    int b = __ldg(start + a), e = __ldg(end + last);
    if (b < 0) {
        b = __ldg(start + a + 1);
        if (b < 0) b = __ldg(start + last);
    }
    if (e < 0) {
        e = __ldg(end + last - 1);
        if (e < 0) e = __ldg(end + a);
    }
    return b >= 0 ? count_run<Ahead>(b, e, pos3, pi, h2) : 0;
}

template <int Ahead>
__global__ void __launch_bounds__(128) k_neighbor_counts_f3(int n, const float *__restrict__ pos3, float cell, int D,
                                                            float h2, const int *__restrict__ start,
                                                            const int *__restrict__ end, int *__restrict__ counts)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *pp = pos3 + 3 * (size_t)i;
    const float3 pi = make_float3(pp[0], pp[1], pp[2]);
    const unsigned m = (unsigned)D - 1u;
    const int cx = cell_coord(pi.x, cell), cy = cell_coord(pi.y, cell), cz = cell_coord(pi.z, cell);
    const unsigned z = (unsigned)cz & m;
    const bool wraps = z == 0u || z == m;
    int cnt = 0;
    // a loop of its own for most warps; not worth its registers with the longer trips (1556 -> 1613 us below)
    if (Ahead == 4 && !__any_sync(__activemask(), wraps)) {
        for (int col = 0; col < 9; ++col)
            cnt += count_cells<Ahead>(cell_addr(cx + col / 3 - 1, cy + col % 3 - 1, cz - 1, D, m), 3, start, end, pos3,
                                      pi, h2);
    } else {  // a warp takes both kinds of column together: each lane its run, then those that wrap the cell left
        const int lo = z == 0u ? 0 : (int)z - 1, alone = z == 0u ? (int)m : 0;
        for (int col = 0; col < 9; ++col) {
            const int base = cell_addr(cx + col / 3 - 1, cy + col % 3 - 1, 0, D, m);
            cnt += count_cells<Ahead>(base + lo, wraps ? 2 : 3, start, end, pos3, pi, h2);
            if (wraps) cnt += count_run<Ahead>(__ldg(start + base + alone), __ldg(end + base + alone), pos3, pi, h2);
        }
    }
    counts[i] = cnt;
}

// Eight positions at a time where cells hold six points on average, and runs
// twice as many as a trip takes (2,000,000 points, a call: 32^3 table, 61 a
// cell, 1637 -> 1556 us, 64^3, 7.6 a cell, 360 -> 352; 128^3, 1.0 a cell, 173
// -> 183; 1,000,003 on 64^3, 3.8 a cell, 106 -> 112).
constexpr long long kDenseCell = 6;

void launch_neighbor_counts_f3(cudaStream_t st, int n, const float *pos3, float cell, int D, float h,
                               const int *start, const int *end, int *counts)
{
    if (n <= 0) return;
    const int grid = (n + 127) / 128;
    if (n >= kDenseCell * D * D * D)
        k_neighbor_counts_f3<8><<<grid, 128, 0, st>>>(n, pos3, cell, D, h * h, start, end, counts);
    else
        k_neighbor_counts_f3<4><<<grid, 128, 0, st>>>(n, pos3, cell, D, h * h, start, end, counts);
}

}  // namespace bp
