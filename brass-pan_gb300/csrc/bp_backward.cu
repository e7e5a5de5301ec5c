// bp_backward.cu -- differentiable rollouts: recording, checkpoints and the
// adjoint driver behind bp_solver_backward.
//
// While a tape is open, every bp_solver_update is recorded (its substep
// constants and parameters) and the state is checkpointed at the start of an
// update once `checkpoint_every` substeps have passed since the last
// checkpoint.  bp_solver_backward walks the recorded substeps backwards: per
// segment between checkpoints it re-runs the forward substeps from the
// checkpoint, keeping each substep's start state, every stage's input
// (SubstepTape) and the grid the substep ran with; then, last substep first,
// it applies the adjoint kernels of the stages in reverse order
// (bp_adjoint.cu).  Each position in a segment has its own buffers, so its
// recording re-run and its adjoint are each captured once as a CUDA graph and
// replayed for every segment.  The neighbour sets of the adjoint walks are those
// of the re-run forward pass.  Finally the solver's state is put back as it
// was before the call.
#include <algorithm>
#include <vector>

#include "bp_solver_state.h"

namespace bp {

// launchers in bp_adjoint.cu
void adj_reorder(cudaStream_t st, const SimConsts &C, const int *order, const float4 *Xprev, const float4 *Vprev,
                 int stabilize, int inv_scaled, const float4 *gP, const float4 *gXs, const float4 *gVs,
                 const float *gW, float4 *gXprev, float4 *gVprev);
void adj_planes(cudaStream_t st, const SimConsts &C, const float4 *Xs, const float4 *Pin, float4 *gP, float4 *gXs);
void adj_commit(cudaStream_t st, int n, float inv_dt, const float4 *gX, const float4 *gV, float4 *gP, float4 *gXs,
                float4 *gVs, float *gW);
void adj_immovable(cudaStream_t st, int k, const int *ids, const int *to_new, float4 *gP, float4 *gXs);
void adj_distance(cudaStream_t st, const DistanceArgs &a, const float4 *Pin, const float *w, const int *to_new,
                  float4 *gP, float *gW, float4 *G1, float4 *G2, float *g_stiff, float *g_rest);
void adj_distance_step(cudaStream_t st, const SimConsts &C, const DistanceStep &a, const float4 *Pin,
                       const float4 *Pplanes, const float4 *gOut, float4 *gIn, float4 *gXs, float *gW, float *g_stiff,
                       float *g_rest);
void adj_wind(cudaStream_t st, const SimConsts &C, const WindArgs &a, const float4 *Pin, const float4 *Vs,
              const float *mass, const int *to_new, float4 *gP, float4 *gVs, float4 *FG, float4 *FV, float4 *FW,
              float4 *g_wind);
void adj_lists(cudaStream_t st, const SimConsts &C, bool record, const float4 *P, const int *off);
void adj_fluid(cudaStream_t st, const SimConsts &C, const float4 *Pin, const float *mass, const float *lam,
               const float *rho, const int *off, const float4 *gOut, const float *gRho, float *gLam, float4 *gPart,
               float4 *GD, float *rhob, float4 *gIn);
void adj_xsph(cudaStream_t st, const SimConsts &C, const float4 *P, const float4 *V, const int *off,
              const float *mass, const float *rho, const float4 *gVout, float4 *gVin, float4 *gX, float *gRho);
void adj_shape_matching(cudaStream_t st, const RigidArgs &a, const float4 *rot, const float4 *Pin, const int *to_new,
                        float4 *gP);
void adj_contacts(cudaStream_t st, const SimConsts &C, const float4 *Pin, const float4 *Xs, const float *w,
                  const int *off, int *count, const float4 *gOut, float4 *gIn, float4 *gXs, float *gW);
void adj_unpick(cudaStream_t st, int id, const int *to_new, float4 *g1, float4 *g2);
void adj_unpick_orig(cudaStream_t st, int n, int id, const int *orig, float4 *g1, float4 *g2);
void adj_bending(cudaStream_t st, const BendingArgs &a, float kb, const float4 *Pin, const float *w, const int *to_new,
                 float4 *gP, float *gW);
void adj_post(cudaStream_t st, const SimConsts &C, const float4 *P, const float4 *V, const float4 *Om,
              const float4 *Nm, const float *rho, const int *off, const float4 *gVb, float4 *gV, float4 *gX,
              float *gRho, float4 *etab, float4 *omb, float4 *ombo, float4 *nmb);

namespace {

// Device buffers owned by a tape (freed with it).
struct DevPool {
    std::vector<std::pair<void *, size_t>> bufs;  // buffer, bytes
    size_t bytes = 0;
    bool failed = false;  // an allocation did
    ~DevPool() { give_back(0); }
    template <class T>
    T *get(size_t count)
    {
        void *p = nullptr;
        const size_t size = std::max<size_t>(count, 1) * sizeof(T);
        if (device_malloc(nullptr, &p, size) != cudaSuccess) {
            failed = true;
            return nullptr;
        }
        bufs.push_back({p, size});
        bytes += size;
        return (T *)p;
    }
    // frees all but the first `count` buffers (those of a set that did not fit)
    void give_back(size_t count)
    {
        for (; bufs.size() > count; bufs.pop_back()) {
            cudaFree(bufs.back().first);
            bytes -= bufs.back().second;
        }
    }
};

// The state a substep starts from.
struct StateBuf {
    float4 *X = nullptr, *V = nullptr, *rot = nullptr, *cm = nullptr;
    int *orig = nullptr;
    int *to_new = nullptr;  // the inverse of orig (picking finds the picked particle through it)
};

// What a substep leaves in the solver's buffers that its adjoint reads: the
// reordered positions, the order and maps, masses, the cell keys and offsets.
struct SubCtx {
    float4 *Xs = nullptr;
    int *order = nullptr, *to_new = nullptr, *keys = nullptr, *off = nullptr;
    float *mass = nullptr, *w = nullptr;
};

}  // namespace

struct Tape {
    int every = 1;
    struct Sub {
        SimConsts C;
        bp_params prm;
        int iterations;
        int ckpt;  // checkpoint taken at the start of this substep, or -1
        // picking (original id, or -1): the target position, and after the
        // last substep of its update (last) the velocity the particle gets
        int picked;
        float3 ppos, pvel;
        bool last;
    };
    std::vector<Sub> subs;
    std::vector<StateBuf> ckpts;  // the first num_ckpts are taken
    int num_ckpts = 0;
    int since = 0;
    StateSnapshot snap;  // the solver's state around backward()
    DevPool pool;
    // per position in a segment: the substep's start state, its stage records,
    // the grid and order it ran with, and the CUDA graphs of its recording
    // re-run and of its adjoint (captured for the configuration in the keys)
    std::vector<StateBuf> seg;
    std::vector<SubstepTape *> tapes;
    std::vector<SubCtx> ctxs;
    std::vector<cudaGraphExec_t> g_fwd, g_bwd;
    std::vector<std::vector<char>> key_fwd, key_bwd, key_warm;
    // adjoint buffers
    bool grads_ready = false;
    float4 *gX = nullptr, *gV = nullptr, *gVn = nullptr, *gP = nullptr, *gP2 = nullptr;
    float4 *gXs = nullptr, *gVs = nullptr, *gPart = nullptr;
    float *gW = nullptr, *gLam = nullptr;
    float4 *G1 = nullptr, *G2 = nullptr, *FG = nullptr, *FV = nullptr, *FW = nullptr, *g_wind = nullptr;
    float *g_stiff = nullptr, *g_rest = nullptr;
    int *contacts = nullptr;  // per particle: its friction contacts (the collision adjoint's pass A)
    // the post passes' adjoint: density gradient (read by the last fluid stage's adjoint), eta-bar,
    // omega-bar of the confinement term, full omega-bar, normal-bar
    float *gRho = nullptr;
    float4 *etab = nullptr, *omb = nullptr, *ombo = nullptr, *nmb = nullptr;
    // the textbook fluid adjoint: (G, D-bar) and rho-bar per particle
    float4 *GD = nullptr;
    float *rhob = nullptr;
};

cudaError_t device_malloc(bp_solver *s, void **p, size_t bytes)
{
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && s && s->spare) {
        cudaStreamSynchronize(s->stream);
        destroy_tape(s->spare);
        s->spare = nullptr;
        cudaGetLastError();
        e = cudaMalloc(p, bytes);
    }
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

void destroy_tape(Tape *t)
{
    if (!t) return;
    for (cudaGraphExec_t g : t->g_fwd)
        if (g) cudaGraphExecDestroy(g);
    for (cudaGraphExec_t g : t->g_bwd)
        if (g) cudaGraphExecDestroy(g);
    for (SubstepTape *st : t->tapes) {
        for (float4 *p : st->pool4) cudaFree(p);
        for (float *p : st->pool1) cudaFree(p);
        delete st;
    }
    delete t;
}

// An optimisation ends and begins a recording for every gradient: allocating
// and freeing the buffers and capturing the graphs again took 4.4 of 11.6 ms
// (128 x 128 flag, 10 frames, on the host while the GPU waits) and 4.8 of
// 11.7 ms (65,536 particles of fluid, 3 frames).  Buffers beyond this many
// bytes are given back at the end of the recording, as those of one that ran
// out of memory are; the kept ones by an end without a recording, where memory
// runs short (device_malloc) and with the solver.
constexpr size_t kSpareTapeBytes = size_t(512) << 20;

void retire_tape(bp_solver *s)
{
    Tape *t = s->tape;
    s->tape = nullptr;
    if (!t) return;
    size_t bytes = t->pool.bytes;
    for (const SubstepTape *st : t->tapes)
        bytes += (st->pool4.size() * sizeof(float4) + st->pool1.size() * sizeof(float)) * (size_t)std::max(s->n, 1);
    for (const auto &b : t->snap.bufs) bytes += b.second;
    bool failed = t->pool.failed || t->snap.copies.size() < t->snap.bufs.size();
    for (const SubstepTape *st : t->tapes) failed = failed || !st->ok;
    if (failed || bytes > kSpareTapeBytes) {
        destroy_tape(t);
        return;
    }
    t->subs.clear();
    t->num_ckpts = 0;
    t->since = 0;
    if (s->spare) destroy_tape(s->spare);
    s->spare = t;
}

int SubstepTape::fresh4()
{
    if (used4 == (int)pool4.size()) {
        void *p = nullptr;
        if (device_malloc(s, &p, (size_t)std::max(s->n, 1) * sizeof(float4)) != cudaSuccess) {
            ok = false;
            return -1;
        }
        pool4.push_back((float4 *)p);
    }
    return used4++;
}

int SubstepTape::snap4(const float4 *src, size_t count)
{
    if (count == 0) count = (size_t)s->n;
    const int slot = fresh4();
    if (slot >= 0)
        cudaMemcpyAsync(pool4[slot], src, count * sizeof(float4), cudaMemcpyDeviceToDevice, s->stream);
    return slot;
}

int SubstepTape::snap1(const float *src)
{
    if (used1 == (int)pool1.size()) {
        void *p = nullptr;
        if (device_malloc(s, &p, (size_t)std::max(s->n, 1) * sizeof(float)) != cudaSuccess) {
            ok = false;
            return -1;
        }
        pool1.push_back((float *)p);
    }
    cudaMemcpyAsync(pool1[used1], src, (size_t)s->n * sizeof(float), cudaMemcpyDeviceToDevice, s->stream);
    return used1++;
}

namespace {

bool alloc_state(Tape &t, const bp_solver *s, StateBuf &b)
{
    const int nb = s->rigid.num_bodies;
    const size_t before = t.pool.bufs.size();
    b.X = t.pool.get<float4>(s->n);
    b.V = t.pool.get<float4>(s->n);
    b.orig = t.pool.get<int>(s->n);
    b.to_new = t.pool.get<int>(s->n);
    b.rot = t.pool.get<float4>(nb);
    b.cm = t.pool.get<float4>(nb);
    const bool ok = b.X && b.V && b.orig && b.to_new && b.rot && b.cm;
    if (!ok) t.pool.give_back(before);
    return ok;
}

void save_state(const bp_solver *s, const StateBuf &b)
{
    const size_t n = (size_t)s->n;
    cudaMemcpyAsync(b.X, s->Xc, n * sizeof(float4), cudaMemcpyDeviceToDevice, s->stream);
    cudaMemcpyAsync(b.V, s->Vc, n * sizeof(float4), cudaMemcpyDeviceToDevice, s->stream);
    cudaMemcpyAsync(b.orig, s->orig_c, n * sizeof(int), cudaMemcpyDeviceToDevice, s->stream);
    cudaMemcpyAsync(b.to_new, s->to_new, n * sizeof(int), cudaMemcpyDeviceToDevice, s->stream);
    if (s->rigid.num_bodies > 0) {
        const size_t nb = (size_t)s->rigid.num_bodies;
        cudaMemcpyAsync(b.rot, s->rigid.rot, nb * sizeof(float4), cudaMemcpyDeviceToDevice, s->stream);
        cudaMemcpyAsync(b.cm, s->rigid.cm, nb * sizeof(float4), cudaMemcpyDeviceToDevice, s->stream);
    }
}

void copy_state(bp_solver *s, const StateBuf &from, float4 *X, float4 *V, int *orig, int *to_new)
{
    const size_t n = (size_t)s->n;
    cudaMemcpyAsync(X, from.X, n * sizeof(float4), cudaMemcpyDeviceToDevice, s->stream);
    cudaMemcpyAsync(V, from.V, n * sizeof(float4), cudaMemcpyDeviceToDevice, s->stream);
    cudaMemcpyAsync(orig, from.orig, n * sizeof(int), cudaMemcpyDeviceToDevice, s->stream);
    cudaMemcpyAsync(to_new, from.to_new, n * sizeof(int), cudaMemcpyDeviceToDevice, s->stream);
}

// The checkpoint c as the start of the segment's first substep.
void load_state(bp_solver *s, const StateBuf &c, const StateBuf &first)
{
    copy_state(s, c, first.X, first.V, first.orig, first.to_new);
    if (s->rigid.num_bodies > 0) {
        const size_t nb = (size_t)s->rigid.num_bodies;
        cudaMemcpyAsync(s->rigid.rot, c.rot, nb * sizeof(float4), cudaMemcpyDeviceToDevice, s->stream);
        cudaMemcpyAsync(s->rigid.cm, c.cm, nb * sizeof(float4), cudaMemcpyDeviceToDevice, s->stream);
    }
}

bool alloc_ctx(Tape &t, const bp_solver *s, SubCtx &c)
{
    const size_t n = (size_t)s->n, before = t.pool.bufs.size();
    c.Xs = t.pool.get<float4>(n);
    c.order = t.pool.get<int>(n);
    c.to_new = t.pool.get<int>(n);
    c.keys = t.pool.get<int>(n);
    c.off = t.pool.get<int>(s->ncells + 1);
    c.mass = t.pool.get<float>(n);
    c.w = t.pool.get<float>(n);
    const bool ok = c.Xs && c.order && c.to_new && c.keys && c.off && c.mass && c.w;
    if (!ok) t.pool.give_back(before);
    return ok;
}

// The solver's buffers that a substep leaves for its adjoint.
void save_ctx(bp_solver *s, const SubCtx &c)
{
    const size_t n = (size_t)s->n;
    auto cp = [&](void *to, const void *from, size_t bytes) {
        cudaMemcpyAsync(to, from, bytes, cudaMemcpyDeviceToDevice, s->stream);
    };
    cp(c.Xs, s->Xs, n * sizeof(float4));
    cp(c.order, s->order, n * sizeof(int));
    cp(c.to_new, s->to_new, n * sizeof(int));
    cp(c.keys, s->sorted_keys, n * sizeof(int));
    cp(c.off, s->off, (s->ncells + 1) * sizeof(int));
    cp(c.mass, s->mass, n * sizeof(float));
    cp(c.w, s->w, n * sizeof(float));
}

// While it lives, the solver works on the buffers of c (and its committed
// state is st, where given) instead of its own: a substep leaves them filled,
// or its adjoint reads them, without a copy.
struct OnBuffers {
    bp_solver *s;
    float4 *Xs, *Vs, *Xc, *Vc;
    int *order, *to_new, *keys, *off, *orig_c;
    float *mass, *w;
    OnBuffers(bp_solver *s_, const SubCtx &c, const StateBuf *st)
        : s(s_), Xs(s->Xs), Vs(s->Vs), Xc(s->Xc), Vc(s->Vc), order(s->order), to_new(s->to_new), keys(s->sorted_keys),
          off(s->off), orig_c(s->orig_c), mass(s->mass), w(s->w)
    {
        s->Xs = c.Xs;
        s->order = c.order;
        s->to_new = c.to_new;
        s->sorted_keys = c.keys;
        s->off = c.off;
        s->mass = c.mass;
        s->w = c.w;
        if (st) {
            s->Xc = st->X;
            s->Vc = st->V;
            s->orig_c = st->orig;
        }
    }
    ~OnBuffers()
    {
        s->Xs = Xs;
        s->Vs = Vs;
        s->Xc = Xc;
        s->Vc = Vc;
        s->order = order;
        s->to_new = to_new;
        s->sorted_keys = keys;
        s->off = off;
        s->orig_c = orig_c;
        s->mass = mass;
        s->w = w;
    }
};

bool stage_on(const bp_params &p, int bit) { return (p.stage_mask & bit) != 0; }

bp_status ensure_grads(Tape &t, const bp_solver *s)
{
    if (t.grads_ready) return BP_OK;
    const size_t n = (size_t)s->n, before = t.pool.bufs.size();
    const size_t m = (size_t)s->dist.num_edges, f = (size_t)s->wind.num_faces;
    t.gX = t.pool.get<float4>(n);
    t.gV = t.pool.get<float4>(n);
    t.gVn = t.pool.get<float4>(n);
    t.gP = t.pool.get<float4>(n);
    t.gP2 = t.pool.get<float4>(n);
    t.gXs = t.pool.get<float4>(n);
    t.gVs = t.pool.get<float4>(n);
    t.gPart = t.pool.get<float4>(n);
    t.gW = t.pool.get<float>(n);
    t.gLam = t.pool.get<float>(n);
    t.G1 = t.pool.get<float4>(m);
    t.G2 = t.pool.get<float4>(m);
    t.FG = t.pool.get<float4>(3 * f);
    t.FV = t.pool.get<float4>(f);
    t.FW = t.pool.get<float4>(f);
    t.g_wind = t.pool.get<float4>(1);
    t.g_stiff = t.pool.get<float>(m);
    t.g_rest = t.pool.get<float>(m);
    t.contacts = t.pool.get<int>(n);
    t.gRho = t.pool.get<float>(n);
    t.etab = t.pool.get<float4>(n);
    t.omb = t.pool.get<float4>(n);
    t.ombo = t.pool.get<float4>(n);
    t.nmb = t.pool.get<float4>(n);
    t.GD = t.pool.get<float4>(n);
    t.rhob = t.pool.get<float>(n);
    if (!(t.gX && t.gV && t.gVn && t.gP && t.gP2 && t.gXs && t.gVs && t.gPart && t.gW && t.gLam && t.G1 &&
          t.G2 && t.FG && t.FV && t.FW && t.g_wind && t.g_stiff && t.g_rest && t.contacts && t.gRho && t.etab &&
          t.omb && t.ombo && t.nmb && t.GD && t.rhob)) {
        t.pool.give_back(before);
        return fail_with(BP_ERR_OUT_OF_MEMORY, "backward: gradient buffers");
    }
    t.grads_ready = true;
    return BP_OK;
}

// The adjoint of one substep whose taped re-run just finished (orig: the
// original id of each sorted particle, as it committed them); (gX, gV) are
// the gradients w.r.t. its committed state on entry and w.r.t. its start
// state (start.X, start.V, in the previous order) on exit.  Both keep their
// buffers (t.gX, t.gV) from substep to substep, so the sequence can be captured
// once and replayed for every substep.
void adjoint_substep(bp_solver *s, Tape &t, const Tape::Sub &u, const StateBuf &start, const int *orig,
                     const SubstepTape &T)
{
    const cudaStream_t st = s->stream;
    SimConsts C = u.C;  // the adjoint walks take the 27 cells, recording their pairs in the list buffer
    C.vl = nullptr;
    C.nl_pos = nullptr;
    C.sl_pos = nullptr;
    C.cell_keys = s->sorted_keys;
    if (C.sl_first) C.sl_first = s->off;
    C.nl_stats = nullptr;
    // nor the alias classes: their class-order positions are gathered only
    // for the forward walks (the same candidates in the same order remain)
    C.cls_perm = nullptr;
    C.cls_post = 0;
    if (!(u.prm.walk_options & BP_WALK_NO_LISTS)) {
        C.nbr = s->nbr;
        C.nbr_count = s->nbr_count;  // the fluid adjoint's pass A leaves its lists for pass B
        C.nbr_cap = s->nbr_cap;
    }
    // One search for the stages that walk (k_adj_record_lists) where the update
    // itself takes its lists so and two of them read them: the density passes,
    // and XSPH alone after the commit (the post passes record their own).
    SimConsts Cl = C;
    bool listed = false;
    int list_passes = 0;
    int readers = 0;
    for (const TapeRec &rec : T.recs) readers += rec.stage == TS_FLUID || rec.stage == TS_XSPH;
    const bool shared = u.C.sl_pos && C.nbr && s->walk_xyz && readers > 1;
    if (shared) {
        Cl.sl_pos = u.C.sl_pos;
        Cl.walk_xyz = s->walk_xyz;
        Cl.walk_stride = s->walk_stride;
    }
    auto lists_at = [&](const float4 *P) -> const SimConsts & {
        if (!shared) return C;
        if (!listed) {
            LaunchLog L;
            launch_walk_planes(st, s->n, P, s->walk_xyz, s->walk_stride, &L);
            clear_list_bits(s);
        }
        Cl.sl_pass = list_passes++ & 1;
        adj_lists(st, Cl, !listed, P, s->off);
        listed = true;
        return Cl;
    };
    const bp_params &p = u.prm;
    const bool planes = stage_on(p, BP_STAGE_PLANES) && s->nplanes > 0;
    const bool distance = stage_on(p, BP_STAGE_DISTANCE) && s->dist.num_edges > 0;
    const bool pcoll = stage_on(p, BP_STAGE_PARTICLE_COLLISION) && s->has_solid;
    const bool bending = stage_on(p, BP_STAGE_BENDING) && s->bend.num_quads > 0;
    // the post passes' and XSPH's density gradient, for the last fluid stage (the density they read)
    cudaMemsetAsync(t.gRho, 0, (size_t)s->n * sizeof(float), st);
    bool last_fluid = true;
    // the gradient of the positions, and of the velocities, as the stages are
    // undone, and the buffer of each that the next one writes
    float4 *gP = t.gP, *gP2 = t.gP2, *gV = t.gV, *gVn = t.gVn;
    // the velocity the update gave the picked particle after its last substep
    if (u.last && u.picked >= 0) adj_unpick(st, u.picked, s->to_new, gV, nullptr);
    for (int r = (int)T.recs.size() - 1; r >= 0; --r) {
        // a cloth iteration's end and the planes directly before it in one launch
        const int imm = T.recs[r].stage == TS_IMMOVABLE ? 1 : 0, d = r - imm;
        if (s->dist_step.range && d >= 0 && T.recs[d].stage == TS_DISTANCE) {
            const bool pl = d > 0 && T.recs[d - 1].stage == TS_PLANES;
            DistanceStep ds = s->dist_step;
            if (!imm) ds.pinned = nullptr;
            ds.orig_s = orig;
            ds.to_new = s->to_new;
            ds.w = s->w;
            ds.Xs = s->Xs;
            adj_distance_step(st, C, ds, T.pool4[T.recs[d].slot], pl ? T.pool4[T.recs[d - 1].slot] : nullptr, gP, gP2,
                              t.gXs, t.gW, t.g_stiff, t.g_rest);
            std::swap(gP, gP2);
            r = pl ? d - 1 : d;
            continue;
        }
        const TapeRec &rec = T.recs[r];
        switch (rec.stage) {
        case TS_POST_AB: {  // positions: the commit's input; velocities before pass A in the slot
            int c = r - 1;
            while (c >= 0 && T.recs[c].stage != TS_COMMIT) --c;
            const float4 *Pc = T.pool4[T.recs[c].slot];
            const float *rho = T.pool1[rec.aux1];
            if (C.use_xsph) {  // pass C first: gV -> the gradient of pass B's velocities
                adj_xsph(st, C, Pc, T.pool4[rec.aux + 2], s->off, s->mass, rho, gV, gVn, t.gX, t.gRho);
                std::swap(gV, gVn);
            }
            adj_post(st, C, Pc, T.pool4[rec.slot], T.pool4[rec.aux], T.pool4[rec.aux + 1], rho, s->off, gV, gVn,
                     t.gX, t.gRho, t.etab, t.omb, t.ombo, t.nmb);
            std::swap(gV, gVn);
            break;
        }
        case TS_PICK:  // the iteration's target position
            adj_unpick(st, u.picked, s->to_new, gP, nullptr);
            break;
        case TS_BENDING:
            adj_bending(st, s->bend, p.bending_stiffness, T.pool4[rec.slot], s->w, s->to_new, gP, t.gW);
            break;
        case TS_XSPH: {  // velocities before XSPH in the slot; positions: the commit's input
            int c = r - 1;
            while (c >= 0 && T.recs[c].stage != TS_COMMIT) --c;
            const float4 *Pc = T.pool4[T.recs[c].slot];
            adj_xsph(st, lists_at(Pc), Pc, T.pool4[rec.slot], s->off, s->mass, T.pool1[rec.aux1], gV,
                     gVn, t.gX, t.gRho);
            std::swap(gV, gVn);
            break;
        }
        case TS_COMMIT:
            adj_commit(st, s->n, C.inv_dt, t.gX, gV, gP, t.gXs, t.gVs, t.gW);
            break;
        case TS_IMMOVABLE:
            adj_immovable(st, s->nimm, s->imm, s->to_new, gP, t.gXs);
            break;
        case TS_DISTANCE:
            adj_distance(st, s->dist, T.pool4[rec.slot], s->w, s->to_new, gP, t.gW, t.G1, t.G2, t.g_stiff,
                         t.g_rest);
            break;
        case TS_FLUID:
            adj_fluid(st, lists_at(T.pool4[rec.slot]), T.pool4[rec.slot], s->mass, T.pool1[rec.aux], T.pool1[rec.aux + 1], s->off, gP,
                      last_fluid ? t.gRho : nullptr, t.gLam, t.gPart, t.GD, t.rhob, gP2);
            last_fluid = false;
            std::swap(gP, gP2);
            break;
        case TS_PLANES:
            adj_planes(st, C, s->Xs, T.pool4[rec.slot], gP, t.gXs);
            break;
        case TS_PCOLL:
            adj_contacts(st, C, T.pool4[rec.slot], s->Xs, s->w, s->off, t.contacts, gP, gP2, t.gXs, t.gW);
            std::swap(gP, gP2);
            break;
        case TS_SHAPE:
            adj_shape_matching(st, s->rigid, T.pool4[rec.aux], T.pool4[rec.slot], s->to_new, gP);
            break;
        case TS_WIND:
            adj_wind(st, C, s->wind, T.pool4[rec.slot], T.pool4[T.vs_slot], s->mass, s->to_new, gP, t.gVs, t.FG,
                     t.FV, t.FW, t.g_wind);
            break;
        default:  // excluded by check_supported
            break;
        }
    }
    const int inv_scaled = (distance || bending || pcoll) ? 1 : 0;  // the stages that read w
    // (gX, gV) were read by the commit's adjoint, the last to need them
    adj_reorder(st, C, s->order, start.X, start.V, planes ? 1 : 0, inv_scaled, gP, t.gXs, t.gVs, t.gW, t.gX, t.gV);
    // the substep began by setting the picked particle's position and velocity
    if (u.picked >= 0) adj_unpick_orig(st, s->n, u.picked, start.orig, t.gX, t.gV);
}

// The bytes a captured substep depends on: its constants, iteration count and
// parameters (buffer pointers inside them are the solver's own, fixed).
std::vector<char> sub_key(const Tape::Sub &u)
{
    const float pick[8] = {(float)u.picked, u.ppos.x, u.ppos.y, u.ppos.z, u.pvel.x, u.pvel.y, u.pvel.z,
                           u.last ? 1.f : 0.f};
    std::vector<char> k(sizeof(SimConsts) + sizeof(int) + sizeof(bp_params) + sizeof(pick));
    char *p = k.data();
    memcpy(p, &u.C, sizeof(SimConsts));
    memcpy(p += sizeof(SimConsts), &u.iterations, sizeof(int));
    memcpy(p += sizeof(int), &u.prm, sizeof(bp_params));
    memcpy(p += sizeof(bp_params), pick, sizeof(pick));
    return k;
}

// Launches the graph of `enqueue` (captured again when the substep differs
// from the captured one).
template <class F>
bp_status replay(bp_solver *s, cudaGraphExec_t &exec, std::vector<char> &key, const Tape::Sub &u, F &&enqueue)
{
    std::vector<char> k = sub_key(u);
    if (!exec || k != key) {
        if (exec) cudaGraphExecDestroy(exec);
        exec = nullptr;
        cudaGraph_t g = nullptr;
        if (cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return BP_ERR_CUDA;
        enqueue();
        if (cudaStreamEndCapture(s->stream, &g) != cudaSuccess) return BP_ERR_CUDA;
        const cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return BP_ERR_CUDA;
        key = k;
    }
    return cudaGraphLaunch(exec, s->stream) == cudaSuccess ? BP_OK : BP_ERR_CUDA;
}

}  // namespace

// Called by bp_solver_update before it enqueues an update while a tape is open.
bp_status tape_record_update(bp_solver *s, int nsub, float dt, int iterations, int picked, float3 ppos, float3 pvel)
{
    Tape &t = *s->tape;
    int ck = -1;
    if (t.subs.empty() || t.since >= t.every) {
        if (t.num_ckpts == (int)t.ckpts.size()) {
            StateBuf b;
            if (!alloc_state(t, s, b)) return fail_with(BP_ERR_OUT_OF_MEMORY, "tape: checkpoint");
            t.ckpts.push_back(b);
        }
        ck = t.num_ckpts++;
        save_state(s, t.ckpts[ck]);
        t.since = 0;
    }
    SimConsts C = make_consts(s, dt / (float)nsub);
    if (picked >= 0) C.sl_pos = nullptr;  // as the update itself (enqueue_update)
    for (int k = 0; k < nsub; ++k)
        t.subs.push_back(Tape::Sub{C, s->prm, iterations, k == 0 ? ck : -1, picked, ppos, pvel, k == nsub - 1});
    t.since += nsub;
    return BP_OK;
}

}  // namespace bp

using namespace bp;

bool bp_solver::tape_empty() const { return !tape || tape->subs.empty(); }

extern "C" bp_status bp_solver_tape_begin(bp_solver *s, int32_t checkpoint_every)
{
    if (!s) return fail_with(BP_ERR_INVALID_ARGUMENT, "solver is NULL");
    if (checkpoint_every <= 0) return fail_with(BP_ERR_INVALID_ARGUMENT, "checkpoint_every must be positive");
    if (s->tape) retire_tape(s);
    s->tape = s->spare ? s->spare : new (std::nothrow) Tape();
    s->spare = nullptr;
    if (!s->tape) return fail_with(BP_ERR_OUT_OF_MEMORY, "tape");
    s->tape->every = checkpoint_every;
    return BP_OK;
}

extern "C" bp_status bp_solver_tape_end(bp_solver *s)
{
    if (!s) return fail_with(BP_ERR_INVALID_ARGUMENT, "solver is NULL");
    if (s->stream) cudaStreamSynchronize(s->stream);
    if (s->tape) {
        retire_tape(s);
    } else {
        destroy_tape(s->spare);
        s->spare = nullptr;
    }
    return BP_OK;
}

extern "C" bp_status bp_solver_backward(bp_solver *s, const float *grad_positions, const float *grad_velocities,
                                        bp_gradients *out)
{
    if (!s || !out) return fail_with(BP_ERR_INVALID_ARGUMENT, "NULL argument");
    if (!s->tape || s->tape->subs.empty()) return fail_with(BP_ERR_INVALID_ARGUMENT, "backward: nothing recorded");
    Tape &t = *s->tape;
    bp_status stt;
    if ((stt = ensure_grads(t, s)) != BP_OK) return stt;
    const cudaStream_t st = s->stream;
    const int n = s->n;
    const size_t N = (size_t)n;
    BP_CUDA_OR_FAIL(cudaStreamSynchronize(st));
    StateSnapshot &snap = t.snap;
    if ((stt = snap.take(s)) != BP_OK) return stt;

    // incoming gradients, original order -> the final state's sorted order
    cudaMemsetAsync(t.gX, 0, N * sizeof(float4), st);
    cudaMemsetAsync(t.gV, 0, N * sizeof(float4), st);
    if (grad_positions) {
        cudaMemcpyAsync(s->staging, grad_positions, N * 12, cudaMemcpyHostToDevice, st);
        launch_scatter_xyz(st, n, s->staging, s->to_new, t.gX);
    }
    if (grad_velocities) {
        cudaMemcpyAsync(s->staging + 3 * N, grad_velocities, N * 12, cudaMemcpyHostToDevice, st);
        launch_scatter_xyz(st, n, s->staging + 3 * N, s->to_new, t.gV);
    }
    cudaMemsetAsync(t.g_stiff, 0, std::max(s->dist.num_edges, 1) * sizeof(float), st);
    cudaMemsetAsync(t.g_rest, 0, std::max(s->dist.num_edges, 1) * sizeof(float), st);
    cudaMemsetAsync(t.g_wind, 0, sizeof(float4), st);

    const bp_params saved_prm = s->prm;
    LaunchLog L;
    L.stream = st;
    auto bail = [&](bp_status e, const char *msg) {
        s->prm = saved_prm;
        snap.restore(s);
        return fail_with(e, msg);
    };
    int seg_end = (int)t.subs.size();
    while (seg_end > 0) {
        int seg_begin = seg_end - 1;
        while (t.subs[seg_begin].ckpt < 0) --seg_begin;  // substep 0 always holds checkpoint 0
        const int len = seg_end - seg_begin;
        // seg[q] is the start of the segment's substep q, so seg[len] its end
        while ((int)t.seg.size() < len + 1) {
            StateBuf b;
            if (!alloc_state(t, s, b)) return bail(BP_ERR_OUT_OF_MEMORY, "backward: segment buffers");
            t.seg.push_back(b);
        }
        while ((int)t.tapes.size() < len) {
            SubCtx c;
            SubstepTape *tp = new (std::nothrow) SubstepTape();
            if (!tp || !alloc_ctx(t, s, c)) {
                delete tp;
                return bail(BP_ERR_OUT_OF_MEMORY, "backward: segment buffers");
            }
            tp->s = s;
            t.ctxs.push_back(c);
            t.tapes.push_back(tp);
            t.g_fwd.push_back(nullptr);
            t.g_bwd.push_back(nullptr);
            t.key_fwd.emplace_back();
            t.key_bwd.emplace_back();
            t.key_warm.emplace_back();
        }
        // forward from the checkpoint, recording every substep: its start
        // state, each stage's input and the grid it ran with
        load_state(s, t.ckpts[t.subs[seg_begin].ckpt], t.seg[0]);
        for (int k = seg_begin; k < seg_end; ++k) {
            const int q = k - seg_begin;
            const Tape::Sub &u = t.subs[k];
            s->prm = u.prm;
            auto body = [&] {
                SubstepTape &T = *t.tapes[q];
                const StateBuf &from = t.seg[q], &to = t.seg[q + 1];
                T.reset();
                SimConsts C = u.C;
                if (u.picked < 0) {  // straight from and into the segment's buffers
                    OnBuffers on(s, t.ctxs[q], &from);
                    T.next_X = to.X;
                    T.next_V = to.V;
                    T.next_orig = to.orig;
                    C.cell_keys = s->sorted_keys;
                    if (C.sl_first) C.sl_first = s->off;
                    enqueue_substep(s, C, u.iterations, u.picked, u.ppos, &L, &T);
                    return;
                }
                // the pick changes the start state in place and finds its
                // particle through the map of the substep before
                copy_state(s, from, s->Xc, s->Vc, s->orig_c, s->to_new);
                if (q > 0)
                    cudaMemcpyAsync(s->to_new, t.ctxs[q - 1].to_new, N * sizeof(int), cudaMemcpyDeviceToDevice, st);
                T.next_X = T.next_V = nullptr;
                T.next_orig = nullptr;
                enqueue_substep(s, C, u.iterations, u.picked, u.ppos, &L, &T);
                if (u.last)  // the end of its update: the picked particle's velocity
                    launch_pick(s->stream, u.picked, s->to_new, s->Xc, u.ppos, 0, s->Vc, u.pvel, &L);
                save_ctx(s, t.ctxs[q]);
                save_state(s, to);
            };
            if (sub_key(u) != t.key_warm[q]) {  // a new configuration runs once directly, growing
                body();                          // the record pool outside any capture
                if (!t.tapes[q]->ok) return bail(BP_ERR_OUT_OF_MEMORY, "backward: stage records");
                t.key_warm[q] = sub_key(u);
            } else {
                const bp_status e = replay(s, t.g_fwd[q], t.key_fwd[q], u, body);
                if (e != BP_OK) return bail(e, "backward: recording graph");
            }
        }
        // last substep first: the adjoint of each, on the grid it ran with
        for (int k = seg_end - 1; k >= seg_begin; --k) {
            const int q = k - seg_begin;
            const Tape::Sub &u = t.subs[k];
            s->prm = u.prm;
            const bp_status e = replay(s, t.g_bwd[q], t.key_bwd[q], u, [&] {
                OnBuffers on(s, t.ctxs[q], nullptr);
                adjoint_substep(s, t, u, t.seg[q], t.seg[q + 1].orig, *t.tapes[q]);
            });
            if (e != BP_OK) return bail(e, "backward: adjoint graph");
        }
        seg_end = seg_begin;
    }
    s->prm = saved_prm;

    // gradients w.r.t. the state at tape_begin, in its order -> original order
    const int *orig0 = t.ckpts[0].orig;
    bp_status result = BP_OK;
    if (out->positions) {
        launch_gather_xyz(st, n, t.gX, orig0, s->staging);
        cudaMemcpyAsync(out->positions, s->staging, N * 12, cudaMemcpyDeviceToHost, st);
    }
    if (out->velocities) {
        launch_gather_xyz(st, n, t.gV, orig0, s->staging + 3 * N);
        cudaMemcpyAsync(out->velocities, s->staging + 3 * N, N * 12, cudaMemcpyDeviceToHost, st);
    }
    const size_t m = (size_t)s->dist.num_edges;
    if (out->distance_stiffness && m)
        cudaMemcpyAsync(out->distance_stiffness, t.g_stiff, m * sizeof(float), cudaMemcpyDeviceToHost, st);
    if (out->distance_rest_length && m)
        cudaMemcpyAsync(out->distance_rest_length, t.g_rest, m * sizeof(float), cudaMemcpyDeviceToHost, st);
    float4 gw = make_float4(0.f, 0.f, 0.f, 0.f);
    cudaMemcpyAsync(&gw, t.g_wind, sizeof(float4), cudaMemcpyDeviceToHost, st);
    snap.restore(s);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) result = fail_with(BP_ERR_CUDA, std::string("backward: ") + cudaGetErrorString(e));
    if (out->wind_velocity) {
        out->wind_velocity[0] = gw.x;
        out->wind_velocity[1] = gw.y;
        out->wind_velocity[2] = gw.z;
    }
    if (result == BP_OK) {
        const cudaError_t le = cudaGetLastError();
        if (le != cudaSuccess) result = fail_with(BP_ERR_CUDA, std::string("backward: ") + cudaGetErrorString(le));
    }
    return result;
}
