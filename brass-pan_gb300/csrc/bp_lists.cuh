// bp_lists.cuh -- substep lists: one neighbour search per substep
// (SimConsts::sl_pos).  What the passes over them share: who may read a list,
// the queue of those that may not, the walk of a queued particle by a whole
// warp, and the skin.
#pragma once

#include <algorithm>

#include "bp_internal.h"
#include "bp_walk.cuh"

namespace bp {

constexpr unsigned kWarp = 0xffffffffu;

// What a pass over the substep lists does: records them (the substep's first
// lambda pass) or reads them (and queues the particles that may not).
enum ListPass { kRecordLists, kReadLists };

// Appends t to a queue (nullptr: only counts it).
__device__ __forceinline__ void append_to(int *count, int *queue, int t)
{
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(m));
    if (!queue) return;
    base = __shfl_sync(m, base, leader);
    queue[base + __popc(m & ((1u << lane) - 1u))] = t;
}

// May the particle of slot t, at pi, read its list in this pass?  Queues it
// where not.
// (fits: its list holds all it should.  walks: where those that something near
// them keeps from it are counted, except in a substep's last pass.)
__device__ __forceinline__ bool reads_substep_list(const SimConsts &C, int t, int i, float3 p, int3 c,
                                                   const GridView &v, bool fits = true, int walks = kSlWalks)
{
    int state = substep_list_state(C, t, i, p, v.base + cell_addr(c.x, c.y, c.z, v.D, v.mask));
    if (state != 0) C.sl_cell[t] = state == 3 ? kListMoved : kListNone;
    else if (!fits) state = 1;
    if (C.nl_stats) atomicAdd(C.nl_stats + state, 1u);
    if (state == 0) return true;
    append_to(C.sl_count + C.sl_pass, C.sl_queue, t);
    if (state == 3) append_to(C.sl_count + (C.sl_adapt ? kSlDisplaced : walks), nullptr, t);
    return false;
}

// In walk mode's last substep: counts the particle of slot t among those that
// something near them would have kept from reading their lists.
__device__ __forceinline__ void note_substep_list(const SimConsts &C, int t, int i, float3 p, int3 c, const GridView &v)
{
    if (!walk_probe(C)) return;
    const int state = substep_list_state(C, t, i, p, v.base + cell_addr(c.x, c.y, c.z, v.D, v.mask));
    if (state == 0) return;
    C.sl_cell[t] = state == 3 ? kListMoved : kListNone;
    if (state == 3) append_to(C.sl_count + (C.sl_adapt ? kSlDisplaced : kSlWalks), nullptr, t);
}

// The candidates that the walk of particle i in cell c meets, but for the cells
// past the table's end (slots: of its own class alone).
__device__ __forceinline__ int walk_candidates(const SimConsts &C, bool slots, int i, int3 c, const GridView &v)
{
    const unsigned m = v.mask, D = (unsigned)v.D, z = min(max((unsigned)c.z & m, 1u), m - 1u);
    const int *__restrict__ off = slots ? C.cls_off + v.base + (size_t)__ldg(C.cls_of + i) * (size_t)C.cls_T : v.off;
    int n = 0;
    for (int col = 0; col < 9; ++col) {
        const unsigned a = ((unsigned)(c.x + col / 3 - 1) & m) * D * D + ((unsigned)(c.y + col % 3 - 1) & m) * D + z;
        n += __ldg(off + a + 2) - __ldg(off + a - 1);
    }
    return n;
}

// Whether the next substep's fluid passes walk (walk mode), from what they would
// cost, in units of a delta-p pass over lists of the pairs alone (1.18 us a pair
// and particle for 314,432 of them): the lists' entries for a pair, sampled as
// they are recorded, times the readers' shares (lambda 0.8, delta-p 1, pass A
// 1.1, B 1.3, C 1.4), and the queued walks, kQueueSearch searches each; or a
// search in each lambda pass and 1.4 in pass A, from the pairs and candidates of
// a particle (measured at 33 to 67 pairs and 216 to 475 candidates: 97 to 177 us).
// Textbook corrections move particles further than the skin in fluid denser than
// at rest, and there the entries of a wide skin and the queue cost more than the
// searches; in reference mode lists win at every density.
// A frame without substep lists, with lists only, with both: 314,432 particles
// squeezed 1.0, 1.1, 1.2 and 1.3 times 1693, 1806, 2499, 3151 us; 1346, 1990,
// 2899, 4861; 1347, 1782, 2435, 3060; 829,440: 4005, 4233, 5865, 7334; 3198, 4415,
// 6510, 11365; 3183, 4376, 5681, 7117.  Twelve frames of 50 bursting scenes 1.00,
// 1.06 and 1.08 times as fast, the slowest 0.85 and 0.98; 210 frames of the mixed
// scene 8.77, 7.93 and 7.80 ms each.
// The ratio is averaged while lists are read, as a burst is over in a few frames;
// walk mode lasts kWalkSubsteps at a time, whose last one counts who would have
// been queued, at a skin that shrinks faster than by the substep (adapt_skin).
constexpr float kQueueSearch = 4.f, kWalkAbove = 1.05f, kListsBelow = 1.0f;
constexpr int kWalkSubsteps = 4;
// False: nothing was counted in this substep.
__device__ __forceinline__ bool choose_mode(const SimConsts &C, float fluid_walks)
{
    int &left = C.sl_count[kSlWalkMode];
    const float sample = (float)C.sl_count[kSlSample], pairs = (float)C.sl_count[kSlPairs];
    const float entries = (float)C.sl_count[kSlEntries], candidates = (float)C.sl_count[kSlCandidates];
    for (int k = kSlSample; k <= kSlCandidates; ++k) C.sl_count[k] = 0;
    if (left > 1) {
        --left;
        return false;
    }
    C.sl_skin[4] = 0.5f * (C.sl_skin[4] + fluid_walks);
    if (!(pairs > 0.f)) {
        left = 0;
        return true;
    }
    const float wider = 1.0f + C.sl_skin[0], volume = wider * wider * wider;
    if (left == 0) C.sl_skin[3] = entries / (pairs * volume);
    const float search = (0.042f * candidates + 1.7f * pairs + 15.f * sample) / pairs * C.sl_search_cost;
    const float lists = C.sl_skin[3] * volume * (1.8f * C.sl_reads + 1.f + 1.1f * C.sl_post_a + C.sl_post_bc) +
                        kQueueSearch * search * C.sl_skin[4];
    const float walks = (1.f + search) * C.sl_reads + 1.f + 1.4f * search * C.sl_post_a + C.sl_post_bc;
    const float ratio = lists / walks;
    C.sl_skin[5] = left > 0 ? ratio : 0.75f * C.sl_skin[5] + 0.25f * fminf(ratio, 1.5f);
    left = C.sl_skin[5] > (left > 0 ? kListsBelow : kWalkAbove) ? kWalkSubsteps : 0;
    return true;
}

// The skin of the next substep's lists, from how many particles the last pass
// over this one's could not read theirs because something near them had moved
// too far.  A list read costs about (1 + skin / h)^3 and a queued walk about
// ten reads, so the break-even lies at a few queued particles in a hundred;
// their share falls steeply with the skin (1M-particle dam break, frame 20:
// 45 % at 0.03 h, 24 % at 0.05 h, 0.6 % at 0.1 h), so it shrinks slowly and
// stays off the last value that was too small, which it forgets slowly too.
// Past kMaxSkin it grows only while a substep's passes go on walking for half
// a particle's worth or more: a spike in one pass, as where a cloth lands, is
// cheaper walked (150k particles with solids: 1730 us a frame, 1800 us wide).
// Squeezed fluid bursting apart, textbook mode, kWideSkin 0.1, 0.15, 0.2 and
// 0.3 of h: 38,850 particles 1031, 909, 853 and 902 us (larger scenes walk there:
// choose_mode).
// The results do not depend on the skin.
constexpr float kWideWalks = 0.5f, kWideRest = 0.05f;
__device__ __forceinline__ void adapt_skin(const SimConsts &C)
{
    if (!C.sl_adapt || blockIdx.x != 0 || threadIdx.x != 0) return;
    const long long moved = C.sl_count[kSlDisplaced];
    const float fluid_walks = (float)(moved + C.sl_count[kSlWalks]) / (float)C.n;
    const bool walked = C.sl_may_walk && C.sl_count[kSlWalkMode] > 0;
    if (C.sl_may_walk && !choose_mode(C, fluid_walks)) return;
    float skin = C.sl_skin[0], bad = C.sl_skin[1] * 0.998f;
    const float walks = 0.5f * (C.sl_skin[2] + fluid_walks + (float)C.sl_count[kSlContactWalks] / (float)C.n);
    const bool wide = skin >= 0.999f * kMaxSkin;
    if (wide && walks > kWideWalks) {
        skin = fminf(skin * 1.3f, kWideSkin);
    } else if (!wide && moved * 25 > C.n) {
        bad = skin;
        skin = fminf(skin * 1.3f, kMaxSkin);
    } else if (wide ? walks < kWideRest : moved * 100 < C.n) {
        skin = fmaxf(skin * (walked ? 0.8f : 0.9f), fmaxf(fminf(bad * 1.15f, skin), kMinSkin));
    }
    C.sl_skin[0] = skin;
    C.sl_skin[1] = bad;
    C.sl_skin[2] = walks;
}

// Records the candidates within sqrt(r2) of slot t's particle (sorted index
// i) into its list, in walk order and its own entry included; returns what
// nbr_count holds (entries | own entry's index or kNoOwnEntry << 16, or -1:
// overflow).
__device__ __forceinline__ int record_substep_list(const SimConsts &C, const float4 *__restrict__ P, bool slots, int t,
                                                   int i, float3 pi, int3 c, float r2, const GridView &v)
{
    ListWriter list(C.nbr, C.nbr_cap, C.n, t);
    int self = kNoOwnEntry;
    const int me = slots ? t : i;
    // the walk planes hold the order this walk reads, except where a particle
    // left the classes' reach after they were written, or without planes
    const int planes = walk_planes_order(C);
    if (planes == (slots ? 2 : 1)) {
        record_walk_planes(planes, pi, r2, v, C, [&](int c0, unsigned bits) {
            const unsigned d = (unsigned)(me - c0);
            if (d < 32u && ((bits >> d) & 1u)) self = list.cnt + __popc(bits & ((1u << d) - 1u));
            list.push_bits(c0, bits);
        });
    } else {
        if (C.nl_stats) atomicAdd(C.nl_stats + 1, 1u);
        auto push = [&](int j, float4) {
            if (j == me) self = list.cnt;
            list.push(j);
        };
        auto test = [&](int, float4 pj) { return len2(pi - f3(pj)) <= r2; };
        if (slots) walk_classes<true, true>(i, c, 0, v, C, test, push);
        else walk_table<true>(c, 0, P, v, nullptr, -1, test, push);
    }
    const int cnt = list.finish(me);
    return cnt < 0 ? -1 : cnt | (self << 16);
}

// ---- walks by a whole warp ----

// The candidates of the 27-cell walk of real cell c, in walk order, 32 at a
// time: chunk(q, p, in) on every lane, q = the lane's candidate and p its
// position (in: it has one).  slots: the class walk (q a class position, read
// from C.cls_pos), else the table walk (q a sorted index, read from P).  Every
// lane of the warp takes part, with the same particle.
// One thread's walk is a serial chain of about 30 dependent loads and 9 loops
// whose length bounds a launch with few walkers; a warp takes a run's
// candidates at once, five runs' loads in flight (32,768-particle dam break,
// 1000 walkers: 59 us a launch with a thread each, 43 us with 8 lanes each,
// whose four groups diverge).  In crowded cells a run's next 32 candidates load
// while the last are taken (mixed scene, fluid 2.5 times as dense: 9.88 -> 9.68
// ms a frame).
template <class F>
__device__ __forceinline__ void warp_walk(const SimConsts &C, bool slots, int3 c, const float4 *__restrict__ P,
                                          const GridView &v, F &&chunk)
{
    constexpr int kAhead = 5;  // runs
    const int lane = threadIdx.x & 31;
    const unsigned m = v.mask, D = (unsigned)v.D;
    const int sh = __ffs(v.D) - 1;
    const unsigned z0 = (unsigned)(c.z - 1) & m, z2 = (unsigned)(c.z + 1) & m;
    const bool wrap = !(z0 < z2);
    const int runs = wrap ? 18 : 9;  // 9 columns, two pieces each where z wraps around the table
    const float4 *__restrict__ src = slots ? C.cls_pos : P;
    int rb = 0, re = 0;  // lane r finds the ends of run r
    if (lane < runs) {
        const int col = wrap ? lane >> 1 : lane, piece = wrap ? lane & 1 : 0;
        const int xr = c.x + col / 3 - 1, yr = c.y + col % 3 - 1;
        const unsigned base = ((unsigned)xr & m) * D * D + ((unsigned)yr & m) * D;
        const unsigned za = piece ? 0u : z0, zb = wrap ? (piece ? z2 : D - 1u) : z2;
        const int *__restrict__ o = v.off + base;
        if (slots) {
            const int zr = piece ? c.z + 1 : c.z - 1;
            const int cls = ((xr >> sh) & 1) | (((yr >> sh) & 1) << 1) | (((zr >> sh) & 1) << 2);
            o = C.cls_off + v.base + (size_t)cls * (size_t)C.cls_T + base;
        }
        rb = __ldg(o + za);
        re = __ldg(o + zb + 1);
    }
#pragma unroll 1
    for (int r = 0; r < runs; r += kAhead) {
        int b[kAhead], e[kAhead];
        float4 p[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            b[u] = __shfl_sync(0xffffffffu, rb, r + u);  // lanes past the last run hold an empty one
            e[u] = __shfl_sync(0xffffffffu, re, r + u);
            p[u] = b[u] + lane < e[u] ? src[b[u] + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
#pragma unroll 1
            for (int q = b[u] + lane; q - lane < e[u]; q += 32) {
                const float4 next = q + 32 < e[u] ? src[q + 32] : make_float4(0.f, 0.f, 0.f, 0.f);
                chunk(q, p[u], q < e[u]);
                p[u] = next;
            }
    }
}

// The solids among the candidates of the table walk of cell c, in walk order, 32
// at a time as warp_walk's: prefix[j] solids lie before sorted index j, list
// holds theirs.
template <class F>
__device__ __forceinline__ void warp_walk_solids(int3 c, const float4 *__restrict__ P, const GridView &v,
                                                 const int *__restrict__ prefix, const int *__restrict__ list, F &&chunk)
{
    const int lane = threadIdx.x & 31;
    const unsigned m = v.mask, D = (unsigned)v.D;
    const unsigned z0 = (unsigned)(c.z - 1) & m, z2 = (unsigned)(c.z + 1) & m;
    const bool wrap = !(z0 < z2);
    const int runs = wrap ? 18 : 9;
    int rb = 0, re = 0;  // lane r finds the ends of run r
    if (lane < runs) {
        const int col = wrap ? lane >> 1 : lane, piece = wrap ? lane & 1 : 0;
        const unsigned base = ((unsigned)(c.x + col / 3 - 1) & m) * D * D + ((unsigned)(c.y + col % 3 - 1) & m) * D;
        rb = __ldg(prefix + __ldg(v.off + base + (piece ? 0u : z0)));
        re = __ldg(prefix + __ldg(v.off + base + (wrap ? (piece ? z2 : D - 1u) : z2) + 1));
    }
    // mostly few in all: the runs' solids in one sequence, 32 at a time (six queues
    // of the mixed scene's frame, a run after another 336 us, in sequence 330, all
    // candidates 315, as most queued there are cloth; of its late frame, 360 us for
    // all candidates and 345)
    int upto = re - rb;  // solids in the runs up to this lane's
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += t;
    }
    const int total = __shfl_sync(0xffffffffu, upto, 31), first = rb - (upto - (re - rb));
#pragma unroll 1
    for (int k = lane; k - lane < total; k += 32) {
        int r = 0;
#pragma unroll 1
        for (int u = 0; u < runs; ++u) r += k >= __shfl_sync(0xffffffffu, upto, u) ? 1 : 0;
        const int at = k + __shfl_sync(0xffffffffu, first, r & 31);
        const int q = k < total ? __ldg(list + at) : 0;
        chunk(q, k < total ? P[q] : make_float4(0.f, 0.f, 0.f, 0.f), k < total);
    }
}

// Sums of up to kWarpTerms quantities over a warp walk's pairs, in walk order:
// lane c adds quantity c of each pair of a chunk from a row in shared memory
// (a load and an add a pair for all of them together, instead of a shuffle a
// quantity).
constexpr int kWarpTerms = 7;  // odd: a warp's rows fall into different banks
using WarpRows = float[32][kWarpTerms];
// The lanes of `take` add value[0..N) to acc of lanes 0..N, in lane order;
// lanes From and up add scale * value with one rounding.
template <int N, int From = N>
__device__ __forceinline__ void warp_add(WarpRows &rows, unsigned take, const float (&value)[N], float scale, float &acc)
{
    constexpr bool Scaled = From < N;
    static_assert(N + (Scaled ? 1 : 0) <= kWarpTerms, "a row holds kWarpTerms quantities");
    const int lane = threadIdx.x & 31;
    if ((take >> lane) & 1u) {
        float *row = rows[__popc(take & ((1u << lane) - 1u))];
#pragma unroll
        for (int k = 0; k < N; ++k) row[k] = value[k];
        if (Scaled) row[N] = scale;
    }
    __syncwarp();
    if (lane < N) {
        const int n = __popc(take);
#pragma unroll 4
        for (int r = 0; r < n; ++r)
            acc = (Scaled && lane >= From) ? __fmaf_rn(rows[r][N], rows[r][lane], acc) : __fadd_rn(acc, rows[r][lane]);
    }
    __syncwarp();
}

// The candidates of the 27-cell walk of real cell c that pass test(q, p), in
// walk order, in batches of up to 32: batch(k0, n, q, p) on every lane, the
// lanes below n holding hits k0 + lane.  Hits collect in shared memory until a
// batch is full, so that what batch() gathers for them is one round of loads
// for 32 hits instead of one for each run (mixed scene of 150k particles, 13k
// walkers: 28 us a launch with a gather per run).
struct WarpHits {
    float4 p[64];
    int q[64];
};
template <class W, class T, class B>
__device__ __forceinline__ int warp_collect(WarpHits &buf, W &&walk, T &&test, B &&batch)
{
    const int lane = threadIdx.x & 31;
    int done = 0, held = 0;
    walk([&](int q, float4 p, bool in) {
        const bool hit = in && test(q, p);
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        if (!hits) return;
        if (hit) {
            const int k = held + __popc(hits & ((1u << lane) - 1u));
            buf.p[k] = p;
            buf.q[k] = q;
        }
        held += __popc(hits);
        __syncwarp();
        if (held < 32) return;
        batch(done, 32, buf.q[lane], buf.p[lane]);
        done += 32;
        held -= 32;
        const float4 rp = buf.p[32 + lane];
        const int rq = buf.q[32 + lane];
        __syncwarp();
        buf.p[lane] = rp;
        buf.q[lane] = rq;
        __syncwarp();
    });
    if (held) batch(done, held, buf.q[lane], buf.p[lane]);
    __syncwarp();
    return done + held;
}
template <class T, class B>
__device__ __forceinline__ int warp_neighbors(const SimConsts &C, bool slots, int3 c, const float4 *__restrict__ P,
                                              const GridView &v, WarpHits &buf, T &&test, B &&batch)
{
    return warp_collect(buf, [&](auto &&chunk) { warp_walk(C, slots, c, P, v, chunk); }, test, batch);
}

// Writes entry k of slot t's list (layout of ListWriter) where it fits.
__device__ __forceinline__ void put_entry(const SimConsts &C, int t, int k, int q)
{
    if (k < C.nbr_cap) C.nbr[((size_t)(k >> 2) * C.n + t) * 4 + (k & 3)] = q;
}
// Fills up the last record of a list of cnt entries (ListWriter::finish(pad)).
__device__ __forceinline__ void warp_pad(const SimConsts &C, int t, int cnt, int pad)
{
    const int k = cnt + (threadIdx.x & 31);
    if ((cnt & 3) && k < ((cnt + 3) & ~3) && k < C.nbr_cap) C.nbr[((size_t)(k >> 2) * C.n + t) * 4 + (k & 3)] = pad;
}

// CTAs of `threads` for a launch over the queue, a warp per entry, whose length
// only the device knows.  32 of them an SM: walks differ tenfold in length, and
// CTAs that start as others end even that out, where 8 resident ones that each
// took every 8th share left SMs idle (mixed scene 6098 -> 6002 us a frame, 200
// frames in 15.4 -> 14.9 ms; 16: 6043 us and 15.0 ms, 64 as 32); CTAs that find
// no entry cost nothing measurable (1M fluid 4112 and 4121 us).
inline int queue_blocks(int n, int threads)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int per = threads / 32;
    return std::min((n + per - 1) / per, std::max(sms, 1) * 32);
}

}  // namespace bp
