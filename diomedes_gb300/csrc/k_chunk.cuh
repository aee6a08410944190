// k_chunk.cuh -- the whole AVBD solve of a step in one launch: one cluster of
// CTAs per chunk of consecutive scenes, poses resident in shared memory.
//
// The reference dispatches init, then (primal, dual) x iterations, then
// recover as separate compute passes over every body and contact
// (engine/src/render/gpu_physics.rs:541-550), so every iteration re-reads
// every pose and row.  Scenes never couple -- rows and joints stay inside a
// scene -- so a chunk of whole scenes can run its whole schedule alone: its
// snapshot / new poses (both Jacobi parities) and step-start poses live in
// the shared memory of the cluster's CTAs, the phases are separated by
// cluster barriers, and only the rows, joint views and per-body constants
// stream from L1 / L2 / HBM.  Each phase evaluates exactly the expressions of
// the per-phase kernels, so the result is bit-identical to init, 10 x
// (primal, dual), recover launched one by one.
//
// A chunk's bodies are dealt to its CTAs in blocks of 2^blk consecutive
// bodies, round robin: chains and nearby boxes stay in one CTA for the most
// part (their poses are read from its own shared memory, others' through
// distributed shared memory), and a scene's loose boxes, which carry the
// contact rows and follow its chains, are spread over all of them.  Rows are
// dealt evenly for the dual.  One CTA for the whole chunk (the layout before)
// bounded a step by its largest scene: 2,000 bodies are four rounds of 512
// threads an iteration, whatever else the GPU has free; and a CTA that fills
// an SM leaves it idle at every barrier.
#pragma once

#include "k_avbd.cuh"
#include "k_color.cuh"

namespace dio {

// Spread: a cluster of 256-thread CTAs a chunk, two CTAs an SM at 128
// registers (FP64: one), rows staged (grouped primal).  Packed, for worlds
// that fill the GPU several times over: one CTA a chunk, 512 threads (FP64
// 256), the whole SM; a __syncthreads between phases keeps L1, which a
// cluster barrier's acquire empties (measured: a dependent load after it
// takes 266 cycles against 38, the barrier itself 500 cycles, 1,100-1,600
// with a global store in flight).
template <class R, bool kSpread>
__host__ __device__ constexpr int chunk_threads() {
    return sizeof(R) == 4 && !kSpread ? 512 : 256;
}
constexpr uint32_t kMaxClusterShift = 3;  // up to 8 CTAs (the portable cluster size)

// Poses of a chunk in its CTAs' shared memory.  Every body a chunk's rows and
// joints touch lies in the chunk (rows and joints never cross scenes).  With
// one pose type: both pose buffers and the step start, displacements formed
// here.  Split (P wider than R): what other bodies read -- positions, R
// rotations and displacements, per buffer; a body's own P rotation and step
// start stay in global memory.
template <class P, class R>
struct ChunkPoses {
    static constexpr bool kSplit = sizeof(P) != sizeof(R);
    // buffer b of an array at b * step
    A4<P>* pos;
    A4<P>* rot;
    A4<P>* ipos;
    A4<P>* irot;
    A4<R>* rot_r;
    A4<R>* moved_l;
    V2<R>* moved_a;
    uint32_t step;
    // bytes a body; buffers: 2, or 1 in place (buffer 1 is buffer 0)
    __host__ __device__ static constexpr size_t body_bytes(int buffers) {
        return kSplit ? buffers * (sizeof(A4<P>) + 2 * sizeof(A4<R>) + sizeof(V2<R>))
                      : (2 * buffers + 2) * sizeof(A4<P>);
    }
    // lays the arrays out from `base`; returns what follows them
    __device__ __forceinline__ unsigned char* place(unsigned char* base, uint32_t cap, uint32_t buffers) {
        auto take = [&](auto*& p, uint32_t n) {
            p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base);
            base += (size_t)n * cap * sizeof(*p);
        };
        step = buffers > 1u ? cap : 0u;
        take(pos, buffers);
        if constexpr (kSplit) {
            take(rot_r, buffers);
            take(moved_l, buffers);
            take(moved_a, buffers);
        } else {
            take(rot, buffers);
            take(ipos, 1u);
            take(irot, 1u);
        }
        return base;
    }
    __device__ __forceinline__ void put_moved(uint32_t at, const Moved<R>& m) const {
        rot_r[at] = packq(m.q);
        moved_l[at] = pack(m.dl, m.da.x);
        moved_a[at] = V2<R>{m.da.y, m.da.z};
    }
};
// shared memory of a CTA holding `cap` bodies: the poses (spread: then each
// warp's staging of the grouped primal), and the groups' first bodies
template <class R>
__host__ __device__ constexpr size_t spread_stage_words() {
    return chunk_threads<R, true>() / 32 * primal_group_words<R>();
}
template <class P, class R, bool kSpread>
__host__ __device__ constexpr size_t chunk_smem_bytes(uint32_t cap) {
    return cap * ChunkPoses<P, R>::body_bytes(2) + (kSpread ? spread_stage_words<R>() * sizeof(R) : 0) + (size_t)cap * 2;
}
// coloured: one pose buffer (the sweeps are in place), colour, order and
// selection arrays
template <class P, class R, bool kSpread>
__host__ __device__ constexpr size_t chunk_colored_smem_bytes(uint32_t cap) {
    return cap * ChunkPoses<P, R>::body_bytes(1) + (kSpread ? spread_stage_words<R>() * sizeof(R) : 0) + (size_t)cap * 12 +
           (size_t)2 * (kMaxColors + 1) * 4;
}
// bodies of a chunk over all its CTAs, and of a CTA at most
constexpr uint32_t kSolveChunkCap = 2048;
template <class P, bool kSpread>
__host__ __device__ constexpr uint32_t solve_cta_cap() {
    return (sizeof(P) == 4 ? 2048u : 1024u) / (kSpread ? 2u : 1u);
}
template <class P, class R, bool kSpread>
constexpr bool chunk_fits() {
    return chunk_smem_bytes<P, R, kSpread>(solve_cta_cap<P, kSpread>()) <= 227u * 1024u &&
           chunk_colored_smem_bytes<P, R, kSpread>(solve_cta_cap<P, kSpread>()) <= 227u * 1024u &&
           (solve_cta_cap<P, kSpread>() << kMaxClusterShift) >= kSolveChunkCap &&
           solve_cta_cap<P, kSpread>() <= 4u * chunk_threads<R, kSpread>();  // cta_scan4
}
static_assert(chunk_fits<float, float, true>() && chunk_fits<float, float, false>() &&
                  chunk_fits<double, float, true>() && chunk_fits<double, float, false>() &&
                  chunk_fits<double, double, true>() && chunk_fits<double, double, false>(),
              "scene-chunk poses must fit the CTAs' shared memory");

// How a chunk is dealt: 2^cl CTAs, blocks of 2^blk bodies.
struct SolveShape {
    uint32_t cl, blk;
    __host__ __device__ uint32_t owner(uint32_t d) const { return (d >> blk) & ((1u << cl) - 1u); }
    __host__ __device__ uint32_t slot(uint32_t d) const {
        return ((d >> (blk + cl)) << blk) | (d & ((1u << blk) - 1u));
    }
    // chunk position of slot s of CTA `rank`
    __host__ __device__ uint32_t body(uint32_t s, uint32_t rank) const {
        return ((s >> blk) << (blk + cl)) | (rank << blk) | (s & ((1u << blk) - 1u));
    }
    // slots of a CTA of a chunk of nb bodies
    __host__ __device__ uint32_t slots(uint32_t nb) const {
        return ((nb + (1u << (blk + cl)) - 1u) >> (blk + cl)) << blk;
    }
};

__device__ __forceinline__ uint32_t cta_smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// another CTA's shared memory at the address that p has in this CTA
__device__ __forceinline__ uint32_t peer_addr(const void* p, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(cta_smem_addr(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ A4<float> peer_load(const A4<float>* p, uint32_t rank) {
    A4<float> v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(peer_addr(p, rank)));
    return v;
}
__device__ __forceinline__ A4<double> peer_load(const A4<double>* p, uint32_t rank) {
    A4<double> v;
    const uint32_t a = peer_addr(p, rank);
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.z), "=d"(v.w) : "r"(a + 16u));
    return v;
}
__device__ __forceinline__ V2<float> peer_load(const V2<float>* p, uint32_t rank) {
    V2<float> v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(peer_addr(p, rank)));
    return v;
}
__device__ __forceinline__ uint32_t peer_load(const uint32_t* p, uint32_t rank) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer_addr(p, rank)));
    return v;
}
// barrier over the chunk's CTAs; orders their shared and global memory (the
// rows' duals are written by one CTA and read by others)
template <bool kCluster>
__device__ __forceinline__ void chunk_sync() {
    if constexpr (kCluster) {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    } else {
        __syncthreads();
    }
}

template <class P, class R, bool kCluster>
struct ChunkFetch {
    static constexpr bool kSplit = ChunkPoses<P, R>::kSplit;
    const DevWorld<P, R>& w;
    const ChunkPoses<P, R>& c;
    uint32_t rd, wr;  // snapshot and output buffer, as offsets
    uint32_t lo, rank;
    SolveShape shape;
    // a bit per group of bodies: one of its systems has failed solve6's one test
    uint32_t* failed = nullptr;
    uint32_t group = 0;
    __device__ __forceinline__ bool careful() const { return (failed[group >> 5] >> (group & 31u)) & 1u; }
    __device__ __forceinline__ void be_careful() const { atomicOr(&failed[group >> 5], 1u << (group & 31u)); }
    template <class T>
    __device__ __forceinline__ T get(const T* a, uint32_t j) const {
        const uint32_t d = j - lo;
        if constexpr (kCluster) {
            const uint32_t own = shape.owner(d), s = shape.slot(d);
            return own == rank ? a[s] : peer_load(a + s, own);
        } else {
            return a[d];
        }
    }
    __device__ __forceinline__ uint32_t slot(uint32_t i) const { return kCluster ? shape.slot(i - lo) : i - lo; }
    __device__ __forceinline__ A4<P> pos(uint32_t j) const { return get(c.pos + rd, j); }
    __device__ __forceinline__ A4<P> rot(uint32_t i) const {  // a body of this CTA
        if constexpr (kSplit)
            return w.rot[0][i];
        else
            return c.rot[rd + slot(i)];
    }
    __device__ __forceinline__ Q4<R> rot_r(uint32_t j) const {
        if constexpr (kSplit)
            return quat(get(c.rot_r + rd, j));
        else
            return quat(get(c.rot + rd, j));
    }
    __device__ __forceinline__ Moved<R> moved(uint32_t j) const {
        if constexpr (kSplit)
            return moved_of(get(c.rot_r + rd, j), get(c.moved_l + rd, j), get(c.moved_a + rd, j));
        else
            return moved_from<R>(get(c.pos + rd, j), quat(get(c.rot + rd, j)), get(c.ipos, j), get(c.irot, j));
    }
    __device__ __forceinline__ void store(uint32_t i, A4<P> p, A4<P> q) const {  // a body of this CTA
        const uint32_t at = wr + slot(i);
        c.pos[at] = p;
        if constexpr (kSplit) {
            w.rot[0][i] = q;
            c.put_moved(at, moved_from<R>(p, narrowq<R>(quat(q)), w.init_pos[i], w.init_rot[i]));
        } else {
            c.rot[at] = q;
        }
    }
    // avbd_init's result for slot s; buffer 1 holds the step start, read for
    // static bodies and without any iteration
    __device__ __forceinline__ void put(uint32_t i, uint32_t s, const InitPose<P>& p) const {
        if (c.step) c.pos[c.step + s] = p.start_pos;
        c.pos[s] = p.pos;
        if constexpr (kSplit) {
            w.rot[0][i] = p.rot;
            w.init_pos[i] = p.start_pos;
            w.init_rot[i] = p.start_rot;
            const Moved<R> m = moved_from<R>(p.pos, narrowq<R>(quat(p.rot)), p.start_pos, p.start_rot);
            if (c.step) c.put_moved(c.step + s, m);
            c.put_moved(s, m);
        } else {
            if (c.step) c.rot[c.step + s] = p.start_rot;
            c.rot[s] = p.rot;
            c.ipos[s] = p.start_pos;
            c.irot[s] = p.start_rot;
        }
    }
    // the step-start pose of a body of this CTA
    __device__ __forceinline__ A4<P> ipos(uint32_t i) const {
        if constexpr (kSplit)
            return w.init_pos[i];
        else
            return c.ipos[slot(i)];
    }
    __device__ __forceinline__ A4<P> irot(uint32_t i) const {
        if constexpr (kSplit)
            return w.init_rot[i];
        else
            return c.irot[slot(i)];
    }
    // avbd_recover, then the final pose (buffer offset `fin`) into global buffer 0
    __device__ __forceinline__ void recover(uint32_t i, uint32_t fin, const SolveParams<R>& o) const {
        recover_body_f(w, i, *this, o);
        w.pos[0][i] = c.pos[fin + slot(i)];
        if constexpr (kSplit) {
            // without an iteration the two buffers' schedule leaves the pose before
            // the warm start, the in-place one the warm start itself
            if (c.step && o.iterations == 0) w.rot[0][i] = w.init_rot[i];
        } else {
            w.rot[0][i] = c.rot[fin + slot(i)];
        }
    }
};

// First index r in [s0, s1) with ab[r].x >= key (ab sorted by .x there), or
// s1; one warp, 32-way search (every lane must call it).
__device__ __forceinline__ uint32_t warp_lower_bound(const uint2* ab, uint32_t s0, uint32_t s1, uint32_t key) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = s0, hi = s1;  // the answer lies in [lo, hi]
    while (hi - lo > 32) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t probe = lo + lane * step;
        const bool less = probe < hi && ab[probe].x < key;
        const uint32_t k = __popc(__ballot_sync(0xFFFFFFFFu, less));  // probes below key form a prefix
        const uint32_t nlo = k ? lo + (k - 1) * step + 1 : lo;
        const uint32_t nhi = min(hi, lo + k * step);
        lo = nlo;
        hi = nhi;
    }
    const uint32_t probe = lo + lane;
    const bool less = probe < hi && ab[probe].x < key;
    return lo + __popc(__ballot_sync(0xFFFFFFFFu, less));
}

// What a CTA of the solve works on: its chunk's bodies [lo, lo + nb) and its
// run of the dynamic-body list, ordered by work signature (a warp's bodies
// take the same code path).
struct ChunkCta {
    uint32_t lo, nb, rank;
    uint2 dyn;
    // the chunk's rows: a range of the pair-row section (pairs sorted by body
    // a, scenes contiguous) and one of the container section (dynamic bodies
    // in index order)
    uint32_t p0, np, c0, rows;
    __device__ __forceinline__ uint32_t row(uint32_t t) const { return t < np ? p0 + t : c0 + (t - np); }
};
__device__ __forceinline__ ChunkCta chunk_cta(const uint2* chunks, const uint2* dyn_runs, const SceneDesc* scenes,
                                              const SolveShape& shape) {
    ChunkCta c;
    const uint2 ch = chunks[blockIdx.x >> shape.cl];
    c.rank = blockIdx.x & ((1u << shape.cl) - 1u);  // clusters run along x
    c.dyn = dyn_runs[blockIdx.x];
    c.lo = scenes[ch.x].body_lo;
    c.nb = scenes[ch.y - 1].body_hi - c.lo;
    c.p0 = c.np = c.c0 = c.rows = 0;
    return c;
}
// the rows' four bounds, a warp each, into s_rows (read after the next barrier)
__device__ __forceinline__ void chunk_row_bounds(const uint2* ab, const Counters* ctr, const ChunkCta& c,
                                                 uint32_t* s_rows) {
    const uint32_t warp = threadIdx.x >> 5;
    if (warp < 4) {
        const uint32_t m = ctr->rows, split = min(ctr->pair_rows, m);
        const uint32_t r = warp_lower_bound(ab, warp < 2 ? 0u : split, warp < 2 ? split : m,
                                            (warp & 1) ? c.lo + c.nb : c.lo);
        if ((threadIdx.x & 31) == 0) s_rows[warp] = r;
    }
}
__device__ __forceinline__ void take_row_bounds(ChunkCta& c, const uint32_t* s_rows) {
    c.p0 = s_rows[0];
    c.np = s_rows[1] - s_rows[0];
    c.c0 = s_rows[2];
    c.rows = c.np + (s_rows[3] - s_rows[2]);
}

// Exclusive sums of four values a thread (thread-major order) over the CTA;
// returns the total.  s_warp: a word a warp.
__device__ __forceinline__ uint32_t cta_scan4(uint32_t (&v)[4], uint32_t* s_warp) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t mine = v[0] + v[1] + v[2] + v[3];
    uint32_t x = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if (lane >= (uint32_t)off) x += y;
    }
    __syncthreads();
    if (lane == 31u) s_warp[warp] = x;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (uint32_t k = 0; k < blockDim.x / 32u; ++k) {
        if (k < warp) before += s_warp[k];
        total += s_warp[k];
    }
    uint32_t run = before + x - mine;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t t = v[k];
        v[k] = run;
        run += t;
    }
    return total;
}

// The CTA's bodies cut into groups for its warps: at most 32 bodies and
// about `per` incidences -- as few as four when there are warps enough (each
// body's rows are a chain of sums), twice as many until every warp has one
// group.  Bodies without rows are not split up: they fill 32 lanes.  Packed
// CTAs have more groups than warps anyway: 128 incidences, four a body.  The
// cut is made once a step (the rows do not change within it).  first[k]: the
// group's first body, from c.dyn.x; returns the number of groups.
template <bool kSpread, class P, class R>
__device__ __forceinline__ uint32_t chunk_groups(const DevWorld<P, R>& w, const ChunkCta& c, uint16_t* first,
                                                 uint32_t* s_warp) {
    const uint32_t n = c.dyn.y - c.dyn.x, warps = blockDim.x / 32u, u0 = threadIdx.x * 4u;
    uint32_t rows[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) rows[k] = u0 + k < n ? w.solve.rows[c.dyn.x + u0 + k].y : 0u;
    // a body's share of a group in units of 1 / (32 per)
    uint32_t per = kSpread ? 4u : 128u;
    auto share = [&](uint32_t r) { return max(min(r, per) * 32u, per); };
    uint32_t sums[4];
    for (;; per *= 2u) {
#pragma unroll
        for (int k = 0; k < 4; ++k) sums[k] = u0 + k < n ? share(rows[k]) : 0u;
        const uint32_t total = cta_scan4(sums, s_warp);
        if (!kSpread || total <= warps * 32u * per || per >= 4096u) break;
    }
    // a body's group: its sum over 32 per
    uint32_t starts[4], last = 0xFFFFFFFFu;
    if (u0 && u0 <= n) {  // the body before this thread's first
        const uint32_t r = w.solve.rows[c.dyn.x + u0 - 1u].y;
        last = (sums[0] - share(r)) / (32u * per);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        starts[k] = u0 + k < n && sums[k] / (32u * per) != last ? 1u : 0u;
        last = sums[k] / (32u * per);
    }
    uint32_t at[4] = {starts[0], starts[1], starts[2], starts[3]};
    const uint32_t groups = cta_scan4(at, s_warp);
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (starts[k]) first[at[k]] = (uint16_t)(u0 + k);
    return groups;
}

// The primal of `groups` groups by the CTA's warps, taken from the end
// through a shared cursor: the end of a CTA's run holds the bodies without
// joints, whose contact rows make them the longest.  range(k, t, n): group
// k's first position, from t0 on, and bodies.
template <bool kSpread, class P, class R, class F, class S, class Range>
__device__ __forceinline__ void chunk_primal(const DevWorld<P, R>& w, const S& bodies, uint32_t groups, uint32_t t0,
                                             Range&& range, const SolveParams<R>& o, F fetch, R* stage,
                                             uint32_t* cursor) {
    const uint32_t lane = threadIdx.x & 31u;
    for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(cursor, 1u);
        k = __shfl_sync(0xFFFFFFFFu, k, 0);
        if (k >= groups) break;
        uint32_t t, n;
        range(groups - 1u - k, t, n);
        fetch.group = t - t0;
        primal_group<kSpread>(w, bodies, t, n, o, fetch, stage, lane);
    }
}

// avbd_init for the CTA's bodies.  Dynamic bodies leave their constants and
// row lists at their list positions.
template <class P, class R, class F>
__device__ __forceinline__ void chunk_init(const DevWorld<P, R>& w, const ChunkCta& c, const SolveShape& shape,
                                           const SolveParams<R>& o, const F& fetch) {
    for (uint32_t s = threadIdx.x; s < shape.slots(c.nb); s += blockDim.x) {
        const uint32_t d = shape.body(s, c.rank);
        if (d >= c.nb) continue;
        const uint32_t i = c.lo + d;
        if (w.inv[i].w != R(0)) continue;
        InitPose<P> r;
        r.start_pos = r.pos = w.pos[0][i];
        r.start_rot = r.rot = w.rot[0][i];
        r.start_pos.w = P(0);
        fetch.put(i, s, r);
    }
    for (uint32_t t = c.dyn.x + threadIdx.x; t < c.dyn.y; t += blockDim.x) {
        const uint32_t i = w.dyn_list[t];
        fetch.put(i, shape.slot(i - c.lo), init_pose(w, i, t, o));
        const uint32_t j0 = w.row_off[i];
        w.solve.rows[t] = make_uint2(j0, w.row_off[i + 1] - j0);
    }
}

// One cluster per chunk (chunks[c] = scene range [x, y), bodies contiguous;
// dyn_runs[c 2^cl + rank] = a CTA's run of the dynamic-body list).  `cap`:
// bodies a CTA's shared memory holds (the largest chunk's slots).
template <class P, class R, bool kSpread, bool kCluster>
__global__ void __launch_bounds__(chunk_threads<R, kSpread>(), sizeof(R) == 4 && kSpread ? 2 : 1)
    k_solve_chunks(DevWorld<P, R> w, const uint2* chunks, const uint2* dyn_runs, const SceneDesc* scenes, uint32_t cap,
                   SolveShape shape, SolveParams<R> o) {
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    __shared__ uint32_t s_rows[4];
    __shared__ uint32_t s_cursor[2], s_failed[kSolveChunkCap / 32];
    __shared__ uint32_t s_warp[chunk_threads<R, kSpread>() / 32];
    pdl_enter();
    // layout: poses, staging, the groups' first bodies
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    ChunkPoses<P, R> poses;
    R* const stage0 = reinterpret_cast<R*>(poses.place(chunk_smem, cap, 2));
    R* const stage = stage0 + (kSpread ? (tid >> 5) * primal_group_words<R>() : 0);
    uint16_t* const s_first = reinterpret_cast<uint16_t*>(stage0 + (kSpread ? spread_stage_words<R>() : 0));
    ChunkCta c = chunk_cta(chunks, dyn_runs, scenes, shape);
    chunk_row_bounds(w.ab, w.ctr, c, s_rows);
    if (tid < 2) s_cursor[tid] = 0u;
    if (tid < kSolveChunkCap / 32) s_failed[tid] = 0u;
    using Fetch = ChunkFetch<P, R, kCluster>;
    chunk_init(w, c, shape, o, Fetch{w, poses, 0u, cap, c.lo, c.rank, shape});
    chunk_sync<kCluster>();
    take_row_bounds(c, s_rows);
    const uint32_t groups = chunk_groups<kSpread>(w, c, s_first, s_warp);
    __syncthreads();
    auto range = [&](uint32_t k, uint32_t& t, uint32_t& n) {
        const uint32_t u = s_first[k];
        t = c.dyn.x + u;
        n = (k + 1u < groups ? s_first[k + 1u] : c.dyn.y - c.dyn.x) - u;
    };
    for (uint32_t k = 0; k < o.iterations; ++k) {
        const uint32_t rd = (k & 1u) * cap, wr = cap - rd;
        if (tid == 0) s_cursor[(k + 1u) & 1u] = 0u;  // last used before the previous barrier
        chunk_primal<kSpread>(w, ListBodies<P, R>{w}, groups, c.dyn.x, range, o,
                              Fetch{w, poses, rd, wr, c.lo, c.rank, shape, s_failed}, stage, &s_cursor[k & 1u]);
        chunk_sync<kCluster>();
        if (!c.rows) continue;  // the same for all CTAs of the chunk
        const Fetch fd{w, poses, wr, wr, c.lo, c.rank, shape};
        for (uint32_t t = c.rank * nt + tid; t < c.rows; t += nt << shape.cl) dual_row_f(w, c.row(t), fd, o);
        chunk_sync<kCluster>();
    }
    // avbd_recover from the last written buffer (none: the warm start), and
    // the final pose
    const uint32_t rb = (o.iterations & 1u) * cap, fin = o.iterations ? rb : cap;
    const Fetch fr{w, poses, rb, rb, c.lo, c.rank, shape};
    for (uint32_t s = tid; s < shape.slots(c.nb); s += nt) {
        const uint32_t d = shape.body(s, c.rank);
        if (d < c.nb) fr.recover(c.lo + d, fin, o);
    }
}

// ---------------------------------------------------------------------
// The coloured Gauss-Seidel schedule as one launch per step: each chunk
// colours its own dynamic bodies (the Jones-Plassmann rounds of k_color.cuh
// -- priority hash(index), ties by index, smallest colour free among the
// coloured neighbours -- with the colours in shared memory and a barrier
// between a round's selection and its assignment); each CTA sorts its bodies
// by colour, then the chunk runs init, per iteration one in-place primal
// sweep per colour (barrier after each) and the dual, and recover.  One pose
// buffer (the sweeps are in place).  The colouring of a disconnected graph is
// the union of its components' colourings, so per-chunk rounds give the
// colours of the whole-world rounds; results equal the host-driven coloured
// step bit for bit.

// list positions in the order of the colours
template <class P, class R>
struct OrderedBodies {
    static constexpr bool kAhead = false;
    ListBodies<P, R> list;
    const uint32_t* order;
    __device__ __forceinline__ BodyTask<P, R> load(uint32_t k) const { return list.load(order[k]); }
    __device__ __forceinline__ uint32_t joints(uint32_t k, uint32_t i) const { return list.joints(order[k], i); }
    __device__ __forceinline__ JView joint(uint32_t k, uint32_t i, uint32_t q) const {
        return list.joint(order[k], i, q);
    }
};

constexpr uint32_t kChunkColorRounds = 4096;  // Jones-Plassmann rounds before giving up

template <class P, class R, bool kSpread, bool kCluster>
__global__ void __launch_bounds__(chunk_threads<R, kSpread>(), sizeof(R) == 4 && kSpread ? 2 : 1)
    k_solve_chunks_colored(DevWorld<P, R> w, const uint2* chunks, const uint2* dyn_runs, const SceneDesc* scenes,
                           uint32_t cap, SolveShape shape, SolveParams<R> o) {
    extern __shared__ __align__(16) unsigned char chunk_smem[];
    __shared__ uint32_t s_rows[4];
    __shared__ uint32_t s_cursor[2], s_failed[kSolveChunkCap / 32];
    __shared__ uint32_t s_colored, s_ncolors, s_ndyn;
    pdl_enter();
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    ChunkPoses<P, R> poses;
    R* const stage0 = reinterpret_cast<R*>(poses.place(chunk_smem, cap, 1));
    R* const stage = stage0 + (kSpread ? (tid >> 5) * primal_group_words<R>() : 0);
    uint32_t* const s_color =
        reinterpret_cast<uint32_t*>(stage0 + (kSpread ? spread_stage_words<R>() : 0));
    uint32_t* const s_order = s_color + cap;
    uint32_t* const s_sel = s_order + cap;
    uint32_t* const s_cstart = s_sel + cap;  // kMaxColors + 1
    uint32_t* const s_next = s_cstart + kMaxColors + 1;
    ChunkCta c = chunk_cta(chunks, dyn_runs, scenes, shape);
    const uint32_t lo = c.lo, ndyn = c.dyn.y - c.dyn.x, ctas = 1u << shape.cl;
    chunk_row_bounds(w.ab, w.ctr, c, s_rows);
    if (tid == 0) {
        s_colored = 0;
        s_ncolors = 0;
        s_ndyn = ndyn;
    }
    if (tid < kSolveChunkCap / 32) s_failed[tid] = 0u;
    if (tid < 2) s_cursor[tid] = 0u;
    for (uint32_t q = tid; q <= kMaxColors; q += nt) {
        s_cstart[q] = 0;
        s_next[q] = 0;
    }
    // init (the in-place schedule reads and writes one buffer) and colours reset
    const ChunkFetch<P, R, kCluster> f{w, poses, 0u, 0u, lo, c.rank, shape, s_failed};
    chunk_init(w, c, shape, o, f);
    for (uint32_t s = tid; s < shape.slots(c.nb); s += nt) s_color[s] = kNoColor;
    chunk_sync<kCluster>();
    // a value that every CTA of the chunk keeps at the same address, over all of them
    auto over = [&](const uint32_t* v, uint32_t start, auto&& join) {
        uint32_t r = start;
        if constexpr (kCluster)
            for (uint32_t q = 0; q < ctas; ++q) r = join(r, peer_load(v, q));
        else
            r = join(r, *v);
        return r;
    };
    auto sum = [](uint32_t a, uint32_t b) { return a + b; };
    // Jones-Plassmann rounds over the chunk's dynamic bodies
    const uint32_t want = over(&s_ndyn, 0u, sum);
    uint32_t rounds = 0;
    while (over(&s_colored, 0u, sum) < want) {
        if (++rounds > kChunkColorRounds) {
            if (tid == 0) atomicOr(&w.ctr->error_flags, kErrColorOverflow);
            break;
        }
        for (uint32_t t = c.dyn.x + tid; t < c.dyn.y; t += nt) {
            const uint32_t v = w.dyn_list[t], s = shape.slot(v - lo);
            bool sel = false;
            if (s_color[s] == kNoColor) {
                sel = true;
                for_each_neighbour(w, v, [&](uint32_t u) {
                    if (sel && f.get(s_color, u) == kNoColor && !color_beats(v, u)) sel = false;
                });
            }
            s_sel[s] = sel ? 1u : 0u;
        }
        chunk_sync<kCluster>();
        for (uint32_t t = c.dyn.x + tid; t < c.dyn.y; t += nt) {
            const uint32_t v = w.dyn_list[t], s = shape.slot(v - lo);
            if (!s_sel[s]) continue;
            unsigned long long used[kMaxColors / 64] = {0ull, 0ull, 0ull, 0ull};
            for_each_neighbour(w, v, [&](uint32_t u) {
                const uint32_t q = f.get(s_color, u);
                if (q < kMaxColors) used[q >> 6] |= 1ull << (q & 63);
            });
            uint32_t q = kMaxColors;
            for (uint32_t k = 0; k < kMaxColors / 64; ++k)
                if (~used[k]) {
                    q = k * 64 + (__ffsll(~used[k]) - 1);
                    break;
                }
            if (q >= kMaxColors) {
                atomicOr(&w.ctr->error_flags, kErrColorOverflow);
                q = kMaxColors - 1;
            }
            s_color[s] = q;
            atomicAdd(&s_colored, 1u);
            atomicMax(&s_ncolors, q + 1);
        }
        chunk_sync<kCluster>();
    }
    const uint32_t ncolors = over(&s_ncolors, 0u, [](uint32_t a, uint32_t b) { return max(a, b); });
    // colours out, and the CTA's dynamic bodies sorted by colour
    for (uint32_t s = tid; s < shape.slots(c.nb); s += nt) {
        const uint32_t d = shape.body(s, c.rank);
        if (d < c.nb) w.color[lo + d] = s_color[s];
    }
    if (tid == 0) atomicMax(&w.ctr->colors, ncolors);
    for (uint32_t t = c.dyn.x + tid; t < c.dyn.y; t += nt) {
        const uint32_t q = s_color[shape.slot(w.dyn_list[t] - lo)];
        if (q < kMaxColors) atomicAdd(&s_cstart[q + 1], 1u);
    }
    __syncthreads();
    if (tid == 0)
        for (uint32_t q = 0; q < ncolors; ++q) s_cstart[q + 1] += s_cstart[q];
    __syncthreads();
    for (uint32_t t = c.dyn.x + tid; t < c.dyn.y; t += nt) {
        const uint32_t q = s_color[shape.slot(w.dyn_list[t] - lo)];
        if (q < kMaxColors) s_order[s_cstart[q] + atomicAdd(&s_next[q], 1u)] = t;
    }
    __syncthreads();
    take_row_bounds(c, s_rows);
    uint32_t turn = 0;  // alternates the group cursors
    for (uint32_t k = 0; k < o.iterations; ++k) {
        for (uint32_t q = 0; q < ncolors; ++q, turn ^= 1u) {
            if (tid == 0) s_cursor[turn ^ 1u] = 0u;  // last used before the previous barrier
            // groups of 32 bodies, or fewer when the warps would not all get one
            const uint32_t q0 = s_cstart[q], qn = s_cstart[q + 1] - q0;
            uint32_t g = 32;
            while (g > 1 && qn <= (g / 2) * (nt / 32u)) g /= 2;
            auto range = [&](uint32_t e, uint32_t& t, uint32_t& n) {
                t = q0 + e * g;
                n = min(g, qn - e * g);
            };
            chunk_primal<kSpread>(w, OrderedBodies<P, R>{{w}, s_order}, (qn + g - 1) / g, 0u, range, o, f, stage,
                                  &s_cursor[turn]);
            chunk_sync<kCluster>();
        }
        if (!c.rows) continue;  // the same for all CTAs of the chunk
        for (uint32_t t = c.rank * nt + tid; t < c.rows; t += nt << shape.cl) dual_row_f(w, c.row(t), f, o);
        chunk_sync<kCluster>();
    }
    for (uint32_t s = tid; s < shape.slots(c.nb); s += nt) {
        const uint32_t d = shape.body(s, c.rank);
        if (d >= c.nb) continue;
        f.recover(lo + d, 0u, o);
    }
    chunk_sync<kCluster>();  // peers may still be reading this CTA's counts
}

}  // namespace dio
