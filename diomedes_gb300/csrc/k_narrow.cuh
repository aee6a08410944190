// k_narrow.cuh -- narrow phase on sm_103a.
//
// Restates engine/gpu_physics/narrowphase/src/{lib,support,cuboid,gjk,epa}.rs.
// Work split (the reference runs one thread per pair for everything):
//   k_narrow_main  one thread per pair: clears the pair's slots, runs the box
//                  SAT manifold or the analytic sphere test in-thread, and
//                  queues every other pair for GJK.
//   k_gjk          one thread per queued pair: GJK with witness tracking;
//                  intersecting pairs queue their final simplex for EPA.
//   k_epa          one warp per queued pair: the expanding polytope lives in
//                  shared memory; face search, visibility, horizon extraction
//                  and face compaction are lane-parallel with ballot/scan,
//                  preserving the reference's sequential face order exactly.
#pragma once

#include "engine.cuh"

namespace dio {

template <class R>
struct ShapeR {
    uint32_t tag, hf, hc;
    V3<R> c[4];
};

template <class R>
__device__ __forceinline__ ShapeR<R> load_shape(const DioShape* s) {
    ShapeR<R> o;
    const uint4 h = *reinterpret_cast<const uint4*>(s);
    o.tag = h.x;
    o.hf = h.y;
    o.hc = h.z;
    const float4* c = reinterpret_cast<const float4*>(s->corners);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float4 v = c[i];
        o.c[i] = {R(v.x), R(v.y), R(v.z)};
    }
    return o;
}

template <class R>
struct NB {
    V3<R> pos;
    Q4<R> rot;
    ShapeR<R> shape;
};

// The first maximum of dot(vertex, d[k]) over a hull's n > 0 vertices, for N
// directions at once: what scanning the list with a strict comparison finds
// (a NaN product never wins, a NaN first product keeps vertex 0).  Each
// direction keeps four running maxima, over every fourth vertex, so four
// loads and comparisons are in flight instead of one chain of them.
template <int N, class R>
__device__ __forceinline__ void hull_supports(const A4<R>* hull, uint32_t n, const V3<R> (&d)[N], uint32_t (&best)[N]) {
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    R bd[N][4];
    uint32_t bi[N][4];
    const V3<R> v0 = xyz(hull[0]);
    bool first_nan[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const R d0 = dot(v0, d[k]);
        first_nan[k] = isnan(d0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            bd[k][q] = q ? -R(INFINITY) : d0;
            bi[k][q] = q ? kNone : 0u;
        }
    }
    auto visit = [&](uint32_t i, int q) {
        const V3<R> v = xyz(hull[i]);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const R dd = dot(v, d[k]);
            if (dd > bd[k][q]) {
                bd[k][q] = dd;
                bi[k][q] = i;
            }
        }
    };
    uint32_t i = 0;
    for (; i + 4u <= n; i += 4u)
#pragma unroll
        for (int q = 0; q < 4; ++q) visit(i + q, q);
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if (i + q < n) visit(i + q, q);
#pragma unroll
    for (int k = 0; k < N; ++k) {
        R b = bd[k][0];
        uint32_t at = bi[k][0];
#pragma unroll
        for (int q = 1; q < 4; ++q)
            if (bi[k][q] != kNone && (bd[k][q] > b || (bd[k][q] == b && bi[k][q] < at))) {
                b = bd[k][q];
                at = bi[k][q];
            }
        best[k] = first_nan[k] ? 0u : at;
    }
}

// support, support.rs:21-61 (first max wins ties); BOX shares the cube's sign
// select, HULL scans its vertex list with the same first-max rule.
template <class R>
__device__ __forceinline__ V3<R> support(const ShapeR<R>& s, V3<R> d, const A4<R>* hull) {
    switch (s.tag) {
        case DIO_SHAPE_SPHERE:
            return scale(normalize_or_zero(d), s.c[0].x);
        case DIO_SHAPE_CUBE:
        case DIO_SHAPE_BOX:
            return {d.x >= R(0) ? s.c[0].x : -s.c[0].x, d.y >= R(0) ? s.c[0].y : -s.c[0].y,
                    d.z >= R(0) ? s.c[0].z : -s.c[0].z};
        case DIO_SHAPE_TETRAHEDRON: {
            V3<R> best = s.c[0];
            R bd = dot(best, d);
#pragma unroll
            for (int i = 1; i < 4; ++i) {
                R dd = dot(s.c[i], d);
                if (dd > bd) {
                    bd = dd;
                    best = s.c[i];
                }
            }
            return best;
        }
        case DIO_SHAPE_HULL: {
            if (s.hc == 0 || hull == nullptr) return {R(0), R(0), R(0)};
            const V3<R> dirs[1] = {d};
            uint32_t best[1];
            hull_supports<1>(hull + s.hf, s.hc, dirs, best);
            return xyz(hull[s.hf + best[0]]);
        }
        default:
            return {R(0), R(0), R(0)};
    }
}

// Minimum / maximum of the finite values of the lanes with `has`, among the
// lanes of the mask (an aligned group of kLanes), ties to the lowest index: the index (0xFFFFFFFF: no lane has one).  FP32: the
// values as ordered integers through two redux instructions (five rounds of
// two shuffles took ten times as long); -0 is taken as +0, as a comparison
// takes it.
__device__ __forceinline__ uint32_t order_bits(float x) {
    const uint32_t u = __float_as_uint(x + 0.f);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}
template <bool kMax, int kLanes, class R>
__device__ __forceinline__ uint32_t lanes_best(bool has, R v, uint32_t index, uint32_t mask) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    if constexpr (sizeof(R) == 4) {
        // ordered bits of a number lie strictly between 0 and 2^32 - 1
        const uint32_t key = order_bits(v);
        const uint32_t best = kMax ? __reduce_max_sync(mask, has ? key : 0u) : __reduce_min_sync(mask, has ? key : kAll);
        return __reduce_min_sync(mask, has && key == best ? index : kAll);
    } else {
        uint32_t bi = has ? index : kAll;
#pragma unroll
        for (int off = kLanes / 2; off > 0; off >>= 1) {
            const R ov = __shfl_xor_sync(mask, v, off);
            const uint32_t oi = __shfl_xor_sync(mask, bi, off);
            if (oi != kAll && (bi == kAll || (kMax ? ov > v : ov < v) || (ov == v && oi < bi))) {
                v = ov;
                bi = oi;
            }
        }
        return bi;
    }
}
template <bool kMax, class R>
__device__ __forceinline__ uint32_t warp_best(bool has, R v, uint32_t index) {
    return lanes_best<kMax, 32>(has, v, index, 0xFFFFFFFFu);
}

// support() of a hull with the 32 lanes of a warp over its vertices (every
// lane calls it with the same arguments and gets the same vertex): each
// lane keeps its first maximum over vertices lane, lane + 32, ..., then the
// warp keeps the largest value, ties to the lower index -- the first
// maximum in vertex order, as the serial scan finds it (NaN products never
// win a strict comparison there, and a NaN first product keeps vertex 0).
template <class R>
__device__ __forceinline__ V3<R> support_warp(const ShapeR<R>& s, V3<R> d, const A4<R>* hull, uint32_t lane) {
    if (s.tag != DIO_SHAPE_HULL || s.hc == 0 || hull == nullptr) return support(s, d, hull);
    const V3<R> v0 = xyz(hull[s.hf]);
    if (isnan(dot(v0, d))) return v0;
    R bv = R(0);
    uint32_t bi = 0xFFFFFFFFu;
    for (uint32_t i = lane; i < s.hc; i += 32) {
        const R dd = dot(xyz(hull[s.hf + i]), d);
        if (!isnan(dd) && (bi == 0xFFFFFFFFu || dd > bv)) {
            bv = dd;
            bi = i;
        }
    }
    bi = warp_best<true>(bi != 0xFFFFFFFFu, bv, bi);
    return xyz(hull[s.hf + bi]);
}

// The same with an aligned group of kG lanes (mask: theirs); kG = 1: support().
template <int kG, class R>
__device__ __forceinline__ V3<R> support_group(const ShapeR<R>& s, V3<R> d, const A4<R>* hull, uint32_t lane,
                                               uint32_t mask) {
    if (kG == 1 || s.tag != DIO_SHAPE_HULL || s.hc == 0 || hull == nullptr) return support(s, d, hull);
    const V3<R> v0 = xyz(hull[s.hf]);
    if (isnan(dot(v0, d))) return v0;
    R bv = R(0);
    uint32_t bi = 0xFFFFFFFFu;
    for (uint32_t i = lane & (kG - 1); i < s.hc; i += kG) {
        const R dd = dot(xyz(hull[s.hf + i]), d);
        if (!isnan(dd) && (bi == 0xFFFFFFFFu || dd > bv)) {
            bv = dd;
            bi = i;
        }
    }
    bi = lanes_best<true, kG>(bi != 0xFFFFFFFFu, bv, bi, mask);
    return xyz(hull[s.hf + bi]);
}

template <int kG, class R>
__device__ __forceinline__ void support_witness(const NB<R>& a, const NB<R>& b, V3<R> d, const A4<R>* hull,
                                                V3<R>& point, V3<R>& wit, uint32_t lane, uint32_t mask) {
    V3<R> al = rotate(conj(a.rot), d);
    V3<R> ap = add(rotate(a.rot, support_group<kG>(a.shape, al, hull, lane, mask)), a.pos);
    V3<R> bl = rotate(conj(b.rot), neg(d));
    V3<R> bp = add(rotate(b.rot, support_group<kG>(b.shape, bl, hull, lane, mask)), b.pos);
    point = sub(ap, bp);
    wit = ap;
}
// the same with the warp's lanes over hull vertices (all 32 lanes call it)
template <class R>
__device__ __forceinline__ void support_witness_warp(const NB<R>& a, const NB<R>& b, V3<R> d, const A4<R>* hull,
                                                     V3<R>& point, V3<R>& wit, uint32_t lane) {
    V3<R> al = rotate(conj(a.rot), d);
    V3<R> ap = add(rotate(a.rot, support_warp(a.shape, al, hull, lane)), a.pos);
    V3<R> bl = rotate(conj(b.rot), neg(d));
    V3<R> bp = add(rotate(b.rot, support_warp(b.shape, bl, hull, lane)), b.pos);
    point = sub(ap, bp);
    wit = ap;
}

// ---------------------------------------------------------------- SAT
template <class R>
__device__ __forceinline__ void axes_of(Q4<R> q, V3<R> ax[3]) {
    ax[0] = rotate(q, V3<R>{R(1), R(0), R(0)});
    ax[1] = rotate(q, V3<R>{R(0), R(1), R(0)});
    ax[2] = rotate(q, V3<R>{R(0), R(0), R(1)});
}

template <class R>
__device__ __forceinline__ V3<R> box_half(const ShapeR<R>& s) {
    if (s.tag == DIO_SHAPE_BOX) return s.c[0];
    return {s.c[0].x, s.c[0].x, s.c[0].x};
}

// projected radius: cuboid.rs:37-40 for CUBE pairs, per-axis for BOX
template <class R>
__device__ __forceinline__ R box_radius(V3<R> h, const V3<R> ax[3], V3<R> axis, bool per_axis) {
    if (!per_axis) return h.x * (dabs(dot(axis, ax[0])) + dabs(dot(axis, ax[1])) + dabs(dot(axis, ax[2])));
    return h.x * dabs(dot(axis, ax[0])) + h.y * dabs(dot(axis, ax[1])) + h.z * dabs(dot(axis, ax[2]));
}

template <class R>
__device__ __forceinline__ R comp(V3<R> v, uint32_t i) {
    return i == 0 ? v.x : (i == 1 ? v.y : v.z);
}

template <class R>
struct Manifold {
    V3<R> normal;
    R depth;
    V3<R> pa[8], pb[8];
    uint32_t count;
};

// test_axis, cuboid.rs:19-52
template <class R>
__device__ __forceinline__ bool test_axis(V3<R> raw, uint32_t kind, uint32_t index, V3<R> ha, const V3<R> aax[3],
                                          V3<R> hb, const V3<R> bax[3], V3<R> delta, bool per_axis, R& best_ov,
                                          V3<R>& best_n, uint32_t& best_kind, uint32_t& best_idx) {
    if (length_sq(raw) <= R(1.0e-8)) return true;
    V3<R> axis = normalize(raw);
    R ra = box_radius(ha, aax, axis, per_axis);
    R rb = box_radius(hb, bax, axis, per_axis);
    R ov = ra + rb - dabs(dot(delta, axis));
    if (ov < R(0)) return false;
    if (ov < best_ov) {
        best_ov = ov;
        best_n = dot(delta, axis) >= R(0) ? axis : neg(axis);
        best_kind = kind;
        best_idx = index;
    }
    return true;
}

template <class R>
__device__ __forceinline__ void face_frame(V3<R> pos, const V3<R> ax[3], V3<R> h, uint32_t ai, V3<R> outward,
                                           V3<R>* verts, V3<R>& center, V3<R>& u, V3<R>& v, R& eu, R& ev) {
    V3<R> axis = ax[ai];
    V3<R> fn = scale(axis, dot(axis, outward) >= R(0) ? R(1) : R(-1));
    center = add(pos, scale(fn, comp(h, ai)));
    uint32_t ui = ai == 0 ? 1u : 0u;
    uint32_t vi = ai == 2 ? 1u : 2u;
    u = ax[ui];
    v = ax[vi];
    eu = comp(h, ui);
    ev = comp(h, vi);
    if (verts) {
        verts[0] = add(add(center, scale(u, eu)), scale(v, ev));
        verts[1] = add(sub(center, scale(u, eu)), scale(v, ev));
        verts[2] = sub(sub(center, scale(u, eu)), scale(v, ev));
        verts[3] = sub(add(center, scale(u, eu)), scale(v, ev));
    }
}

// clip_plane, cuboid.rs:216-250
template <class R>
__device__ __forceinline__ uint32_t clip_plane(const V3<R>* in, uint32_t n_in, V3<R> normal, R offset, V3<R>* out) {
    if (n_in == 0) return 0;
    uint32_t count = 0;
    V3<R> prev = in[n_in - 1];
    R prev_d = dot(normal, prev) - offset;
    for (uint32_t i = 0; i < n_in; ++i) {
        V3<R> cur = in[i];
        R cur_d = dot(normal, cur) - offset;
        bool pin = prev_d <= R(1.0e-5);
        bool cin = cur_d <= R(1.0e-5);
        if (pin != cin) {
            R den = prev_d - cur_d;
            if (dabs(den) > R(1.0e-8) && count < 8) {
                R t = prev_d / den;
                t = t < R(0) ? R(0) : (t > R(1) ? R(1) : t);
                out[count++] = add(prev, scale(sub(cur, prev), t));
            }
        }
        if (cin && count < 8) out[count++] = cur;
        prev = cur;
        prev_d = cur_d;
    }
    return count;
}

template <class R>
__device__ __forceinline__ void centered_contact(const NB<R>& a, const V3<R> aax[3], V3<R> ha, const NB<R>& b,
                                                 const V3<R> bax[3], V3<R> hb, V3<R> normal, R depth, bool per_axis,
                                                 Manifold<R>& m) {
    R ra = box_radius(ha, aax, normal, per_axis);
    R rb = box_radius(hb, bax, normal, per_axis);
    m.normal = normal;
    m.depth = depth;
    m.pa[0] = add(a.pos, scale(normal, ra));
    m.pb[0] = sub(b.pos, scale(normal, rb));
    m.count = 1;
}

// collide_manifold, cuboid.rs:276-377 (max_contacts 4 = reference, 8 = all)
template <class R>
__device__ bool collide_manifold(const NB<R>& a, const NB<R>& b, uint32_t max_contacts, Manifold<R>& m) {
    bool per_axis = !(a.shape.tag == DIO_SHAPE_CUBE && b.shape.tag == DIO_SHAPE_CUBE);
    V3<R> aax[3], bax[3];
    axes_of(a.rot, aax);
    axes_of(b.rot, bax);
    V3<R> ha = box_half(a.shape), hb = box_half(b.shape);
    V3<R> delta = sub(b.pos, a.pos);
    R best_ov = 3.402823466e+38f;
    if (sizeof(R) == 8) best_ov = R(1.7976931348623157e308);
    V3<R> best_n{R(1), R(0), R(0)};
    uint32_t best_kind = 0, best_idx = 0;
    for (uint32_t i = 0; i < 3; ++i)
        if (!test_axis(aax[i], 0, i, ha, aax, hb, bax, delta, per_axis, best_ov, best_n, best_kind, best_idx))
            return false;
    for (uint32_t i = 0; i < 3; ++i)
        if (!test_axis(bax[i], 1, i, ha, aax, hb, bax, delta, per_axis, best_ov, best_n, best_kind, best_idx))
            return false;
    for (uint32_t i = 0; i < 3; ++i)
        for (uint32_t j = 0; j < 3; ++j)
            if (!test_axis(cross(aax[i], bax[j]), 2, i * 3 + j, ha, aax, hb, bax, delta, per_axis, best_ov, best_n,
                           best_kind, best_idx))
                return false;
    V3<R> normal = best_n;
    R depth = best_ov;
    if (best_kind == 2) {
        centered_contact(a, aax, ha, b, bax, hb, normal, depth, per_axis, m);
        return true;
    }
    bool ref_a = best_kind == 0;
    V3<R> rn = ref_a ? normal : neg(normal);
    // incident_axis, cuboid.rs:198-214
    const V3<R>* iax = ref_a ? bax : aax;
    uint32_t inc_axis = 0;
    R bdot = dabs(dot(iax[0], rn));
    for (uint32_t i = 1; i < 3; ++i) {
        R d = dabs(dot(iax[i], rn));
        if (d > bdot) {
            bdot = d;
            inc_axis = i;
        }
    }
    V3<R> center, u, v, c2, u2, v2;
    R eu, ev, eu2, ev2;
    face_frame(ref_a ? a.pos : b.pos, ref_a ? aax : bax, ref_a ? ha : hb, best_idx, rn, (V3<R>*)nullptr, center, u,
               v, eu, ev);
    V3<R> pa[8], pb[8];
    face_frame(ref_a ? b.pos : a.pos, iax, ref_a ? hb : ha, inc_axis, neg(rn), pa, c2, u2, v2, eu2, ev2);
    uint32_t count = 4;
    count = clip_plane(pa, count, u, dot(u, center) + eu, pb);
    count = clip_plane(pb, count, neg(u), dot(neg(u), center) + eu, pa);
    count = clip_plane(pa, count, v, dot(v, center) + ev, pb);
    count = clip_plane(pb, count, neg(v), dot(neg(v), center) + ev, pa);
    if (count == 0) {
        centered_contact(a, aax, ha, b, bax, hb, normal, depth, per_axis, m);
        return true;
    }
    R ref_plane = dot(rn, center);
    uint32_t cc = 0;
    for (uint32_t i = 0; i < count; ++i) {
        if (cc >= max_contacts) break;
        V3<R> ip = pa[i];
        R pd = ref_plane - dot(rn, ip);
        if (pd < R(-1.0e-5)) continue;
        V3<R> rp = add(ip, scale(rn, pd > R(0) ? pd : R(0)));
        m.pa[cc] = ref_a ? rp : ip;
        m.pb[cc] = ref_a ? ip : rp;
        ++cc;
    }
    if (cc == 0) {
        centered_contact(a, aax, ha, b, bax, hb, normal, depth, per_axis, m);
        return true;
    }
    m.normal = normal;
    m.depth = depth;
    m.count = cc;
    return true;
}

// collide_manifold by an aligned group of eight lanes (mask: theirs, `lane` this
// one's place in it): an axis or two, then a vertex of the clipped polygon, a
// lane.  Same tests on the same values, so the same result: the least overlap
// with the lowest axis on a tie, vertices and contacts at their place in the
// serial order.  The lane with `emit` has contact `at` of `count`.  poly: two
// buffers of eight vertices in shared memory.
constexpr uint32_t kManifoldLanes = 8;
template <class R>
struct GroupContact {
    V3<R> normal, pa, pb;
    R depth;
    uint32_t count, at;
    bool emit;
};
template <class R>
__device__ __forceinline__ V3<R> pick(const V3<R> ax[3], uint32_t i) {
    return i == 0 ? ax[0] : (i == 1 ? ax[1] : ax[2]);
}
template <class R>
__device__ __forceinline__ V3<R> shfl3(uint32_t mask, V3<R> v, uint32_t src) {
    return {__shfl_sync(mask, v.x, (int)src), __shfl_sync(mask, v.y, (int)src), __shfl_sync(mask, v.z, (int)src)};
}
template <class R>
__device__ __forceinline__ void manifold_group(const NB<R>& a, const NB<R>& b, uint32_t max_contacts, uint32_t lane,
                                               uint32_t mask, V3<R> (*poly)[kManifoldLanes], GroupContact<R>& out) {
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    const uint32_t base = (threadIdx.x & 31u) - lane, below = (1u << lane) - 1u;
    out.count = 0;
    out.emit = false;
    const bool per_axis = !(a.shape.tag == DIO_SHAPE_CUBE && b.shape.tag == DIO_SHAPE_CUBE);
    V3<R> aax[3], bax[3];
    axes_of(a.rot, aax);
    axes_of(b.rot, bax);
    const V3<R> ha = box_half(a.shape), hb = box_half(b.shape);
    const V3<R> delta = sub(b.pos, a.pos);
    R best_ov = 3.402823466e+38f;
    if (sizeof(R) == 8) best_ov = R(1.7976931348623157e308);
    V3<R> best_n{R(1), R(0), R(0)};
    uint32_t best_kind = 0, best_t = kNone;
    bool apart = false;
#pragma unroll 1
    for (uint32_t t = lane; t < 15u; t += kManifoldLanes) {
        const uint32_t e = t - 6u;
        const V3<R> raw = t < 3u ? pick(aax, t) : (t < 6u ? pick(bax, t - 3u) : cross(pick(aax, e / 3u), pick(bax, e % 3u)));
        apart = apart || !test_axis(raw, 0u, t, ha, aax, hb, bax, delta, per_axis, best_ov, best_n, best_kind, best_t);
    }
    if (__any_sync(mask, apart)) return;
    const uint32_t t = lanes_best<false, (int)kManifoldLanes>(best_t != kNone, best_ov, best_t, mask);
    const uint32_t owner = base + (t == kNone ? 0u : t & (kManifoldLanes - 1u));  // no axis: the initial values
    const V3<R> normal = shfl3(mask, best_n, owner);
    const R depth = __shfl_sync(mask, best_ov, (int)owner);
    out.normal = normal;
    out.depth = depth;
    auto centered = [&] {
        out.pa = add(a.pos, scale(normal, box_radius(ha, aax, normal, per_axis)));
        out.pb = sub(b.pos, scale(normal, box_radius(hb, bax, normal, per_axis)));
        out.count = 1;
        out.at = 0;
        out.emit = lane == 0;
    };
    if (t != kNone && t >= 6u) {
        centered();
        return;
    }
    const bool ref_a = t == kNone || t < 3u;
    const uint32_t best_idx = t == kNone ? 0u : (ref_a ? t : t - 3u);
    const V3<R> rn = ref_a ? normal : neg(normal);
    V3<R> rax[3], iax[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        rax[k] = ref_a ? aax[k] : bax[k];
        iax[k] = ref_a ? bax[k] : aax[k];
    }
    uint32_t inc_axis = 0;  // incident_axis, cuboid.rs:198-214
    R bdot = dabs(dot(iax[0], rn));
#pragma unroll
    for (uint32_t i = 1; i < 3; ++i) {
        const R d = dabs(dot(iax[i], rn));
        if (d > bdot) {
            bdot = d;
            inc_axis = i;
        }
    }
    V3<R> center, u, v, c2, u2, v2, verts[4];
    R eu, ev, eu2, ev2;
    face_frame(ref_a ? a.pos : b.pos, rax, ref_a ? ha : hb, best_idx, rn, (V3<R>*)nullptr, center, u, v, eu, ev);
    face_frame(ref_a ? b.pos : a.pos, iax, ref_a ? hb : ha, inc_axis, neg(rn), verts, c2, u2, v2, eu2, ev2);
    uint32_t n = 4;
    V3<R> cur = lane == 0 ? verts[0] : (lane == 1 ? verts[1] : (lane == 2 ? verts[2] : verts[3]));
#pragma unroll 1
    for (uint32_t plane = 0; plane < 4u && n; ++plane) {
        const V3<R> axis = plane < 2u ? u : v;
        const V3<R> pn = (plane & 1u) ? neg(axis) : axis;
        const R offset = dot(pn, center) + (plane < 2u ? eu : ev);
        const uint32_t from = base + (lane == 0 ? n - 1u : lane - 1u);
        const R cur_d = dot(pn, cur) - offset;
        const V3<R> prev = shfl3(mask, cur, from);
        const R prev_d = __shfl_sync(mask, cur_d, (int)from);
        const bool live = lane < n, pin = prev_d <= R(1.0e-5), cin = cur_d <= R(1.0e-5);
        const R den = prev_d - cur_d;
        const bool cross_ = live && pin != cin && dabs(den) > R(1.0e-8), keep = live && cin;
        const uint32_t bc = __ballot_sync(mask, cross_) >> base, bk = __ballot_sync(mask, keep) >> base;
        const uint32_t at = (uint32_t)__popc(bc & below) + (uint32_t)__popc(bk & below);
        V3<R>* dst = poly[plane & 1u];
        if (cross_ && at < kManifoldLanes) {
            R s = prev_d / den;
            s = s < R(0) ? R(0) : (s > R(1) ? R(1) : s);
            dst[at] = add(prev, scale(sub(cur, prev), s));
        }
        if (keep && at + (cross_ ? 1u : 0u) < kManifoldLanes) dst[at + (cross_ ? 1u : 0u)] = cur;
        const uint32_t group = (1u << kManifoldLanes) - 1u;
        n = min((uint32_t)__popc(bc & group) + (uint32_t)__popc(bk & group), kManifoldLanes);
        __syncwarp(mask);
        if (lane < n) cur = dst[lane];
    }
    const R pd = dot(rn, center) - dot(rn, cur);
    const uint32_t on = __ballot_sync(mask, lane < n && !(pd < R(-1.0e-5))) >> base;
    const uint32_t all = (uint32_t)__popc(on & ((1u << kManifoldLanes) - 1u));
    if (all == 0) {
        centered();
        return;
    }
    out.count = min(all, max_contacts);
    out.at = (uint32_t)__popc(on & below);
    out.emit = ((on >> lane) & 1u) && out.at < max_contacts;
    const V3<R> rp = add(cur, scale(rn, pd > R(0) ? pd : R(0)));
    out.pa = ref_a ? rp : cur;
    out.pb = ref_a ? cur : rp;
}

// ---------------------------------------------------------------- GJK
template <class R>
struct Simplex {
    V3<R> p[4], w[4];
    uint32_t len;
    __device__ void push_front(V3<R> pt, V3<R> wt) {
#pragma unroll
        for (int i = 3; i > 0; --i)
            if (i <= (int)len) {
                p[i] = p[i - 1];
                w[i] = w[i - 1];
            }
        p[0] = pt;
        w[0] = wt;
        len = len + 1 < 4 ? len + 1 : 4;
    }
    __device__ void remove(uint32_t index) {
#pragma unroll
        for (uint32_t i = 0; i < 3; ++i)
            if (i >= index && i + 1 < len) {
                p[i] = p[i + 1];
                w[i] = w[i + 1];
            }
        len -= 1;
    }
    __device__ void swap12() {
        V3<R> t = p[1];
        p[1] = p[2];
        p[2] = t;
        t = w[1];
        w[1] = w[2];
        w[2] = t;
    }
};

template <class R>
__device__ __forceinline__ bool same_dir(V3<R> a, V3<R> b) { return dot(a, b) > R(0); }
template <class R>
__device__ __forceinline__ V3<R> triple(V3<R> a, V3<R> b, V3<R> c) { return cross(cross(a, b), c); }
template <class R>
__device__ __forceinline__ V3<R> any_perpendicular(V3<R> v) {
    V3<R> axis;
    if (dabs(v.x) <= dabs(v.y) && dabs(v.x) <= dabs(v.z))
        axis = {R(1), R(0), R(0)};
    else if (dabs(v.y) <= dabs(v.z))
        axis = {R(0), R(1), R(0)};
    else
        axis = {R(0), R(0), R(1)};
    return normalize_or_zero(cross(axis, v));
}

// contains_origin, gjk.rs:112-201
template <class R>
__device__ bool contains_origin(Simplex<R>& s, V3<R>& d) {
    if (s.len == 4) {
        V3<R> a = s.p[0];
        V3<R> ao = neg(a), ab = sub(s.p[1], a), ac = sub(s.p[2], a), ad = sub(s.p[3], a);
        V3<R> abc = cross(ab, ac), acd = cross(ac, ad), adb = cross(ad, ab);
        if (same_dir(abc, ao))
            s.remove(3);
        else if (same_dir(acd, ao))
            s.remove(1);
        else if (same_dir(adb, ao))
            s.remove(2);
        else
            return true;
    }
    if (s.len == 1) {
        d = neg(s.p[0]);
        return false;
    }
    if (s.len == 2) {
        V3<R> a = s.p[0];
        V3<R> ab = sub(s.p[1], a), ao = neg(a);
        if (same_dir(ab, ao)) {
            V3<R> t = triple(ab, ao, ab);
            if (length_sq(t) < R(1e-12)) t = any_perpendicular(ab);
            d = t;
        } else {
            s.remove(1);
            d = ao;
        }
        return false;
    }
    if (s.len == 3) {
        V3<R> a = s.p[0];
        V3<R> ab = sub(s.p[1], a), ac = sub(s.p[2], a), ao = neg(a);
        V3<R> abc = cross(ab, ac);
        if (same_dir(cross(abc, ac), ao)) {
            if (same_dir(ac, ao)) {
                s.remove(1);
                d = triple(ac, ao, ac);
            } else if (same_dir(ab, ao)) {
                s.remove(2);
                d = triple(ab, ao, ab);
            } else {
                s.len = 1;
                d = ao;
            }
        } else if (same_dir(cross(ab, abc), ao)) {
            if (same_dir(ab, ao)) {
                s.remove(2);
                d = triple(ab, ao, ab);
            } else {
                s.len = 1;
                d = ao;
            }
        } else {
            if (dot(abc, ao) > R(0)) {
                d = abc;
            } else {
                s.swap12();
                d = neg(abc);
            }
        }
        return false;
    }
    return false;
}

// gjk, gjk.rs:77-109, by an aligned group of kG lanes (mask: theirs; every lane
// the same simplex)
template <int kG, class R>
__device__ bool gjk(const NB<R>& a, const NB<R>& b, const A4<R>* hull, Simplex<R>& s, uint32_t lane, uint32_t mask) {
    V3<R> d = sub(a.pos, b.pos);
    if (d.x == R(0) && d.y == R(0) && d.z == R(0)) d = {R(1), R(0), R(0)};
    s.len = 0;
    V3<R> pt, wt;
    support_witness<kG>(a, b, d, hull, pt, wt, lane, mask);
    s.push_front(pt, wt);
    d = neg(s.p[0]);
    for (int it = 0; it < 64; ++it) {
        support_witness<kG>(a, b, d, hull, pt, wt, lane, mask);
        if (dot(pt, d) < R(0)) return false;
        s.push_front(pt, wt);
        if (contains_origin(s, d)) return true;
        if (length_sq(d) < R(1e-12)) d = any_perpendicular(s.p[0]);
    }
    return false;
}

// ---------------------------------------------------------------- EPA
constexpr int kEpaV = 68;   // 4 simplex points + one per iteration (64)
constexpr int kEpaF = 256;  // face capacity (reference: 512; overflow flagged)
constexpr int kEpaH = 256;  // horizon capacity (reference: 512; overflow flagged)
constexpr int kEpaE = kEpaV * (kEpaV - 1) / 2;  // vertex pairs
template <class R>
__host__ __device__ constexpr int epa_warps() { return sizeof(R) == 8 ? 2 : 4; }  // FP64 polytopes are twice the size

template <class R>
struct EpaSmem {
    A4<R> v[kEpaV];
    A4<R> w[kEpaV];
    A4<R> fnd[kEpaF];      // face normal xyz, distance w
    uint32_t fabc[kEpaF];  // a | b << 8 | c << 16
    uint32_t vis[kEpaF];   // the faces that see the new vertex, in order
    uint32_t hor[kEpaH];   // a | b << 8
    uint32_t edge[(kEpaE + 3) / 4];  // visible faces at each vertex pair (a byte each; zero between uses)
};

__device__ __forceinline__ uint32_t fa_(uint32_t f) { return f & 0xFF; }
__device__ __forceinline__ uint32_t fb_(uint32_t f) { return (f >> 8) & 0xFF; }
__device__ __forceinline__ uint32_t fc_(uint32_t f) { return (f >> 16) & 0xFF; }

// place of the unordered vertex pair (a, b), a != b, in the edge bytes
__device__ __forceinline__ uint32_t edge_at(uint32_t a, uint32_t b) {
    const uint32_t hi = max(a, b), lo = min(a, b);
    return hi * (hi - 1u) / 2u + lo;
}

// add_face arithmetic, epa.rs:58-85.  Returns false for a degenerate face.
template <class R>
__device__ __forceinline__ bool make_face(const EpaSmem<R>& S, uint32_t a, uint32_t b, uint32_t c, A4<R>& nd,
                                          uint32_t& abc) {
    V3<R> va = xyz(S.v[a]);
    V3<R> n = cross(sub(xyz(S.v[b]), va), sub(xyz(S.v[c]), va));
    if (length_sq(n) < R(1e-12)) return false;
    n = normalize(n);
    R dist = dot(n, va);
    if (dist < R(0)) {
        uint32_t t = a;
        a = c;
        c = t;
        n = neg(n);
        dist = -dist;
    }
    nd = pack(n, dist);
    abc = a | (b << 8) | (c << 16);
    return true;
}

// face_contact, epa.rs:193-240
template <class R>
__device__ void face_contact(const EpaSmem<R>& S, A4<R> nd, uint32_t abc, V3<R>& normal, R& depth, V3<R>& pa,
                             V3<R>& pb) {
    uint32_t ia = fa_(abc), ib = fb_(abc), ic = fc_(abc);
    V3<R> va = xyz(S.v[ia]), vb = xyz(S.v[ib]), vc = xyz(S.v[ic]);
    V3<R> n = xyz(nd);
    R dist = nd.w;
    V3<R> closest = scale(n, dist);
    V3<R> v0 = sub(vb, va), v1 = sub(vc, va), v2 = sub(closest, va);
    R d00 = dot(v0, v0), d01 = dot(v0, v1), d11 = dot(v1, v1), d20 = dot(v2, v0), d21 = dot(v2, v1);
    R denom = d00 * d11 - d01 * d01;
    R w1, w2, w3;
    if (dabs(denom) > R(1e-12)) {
        w2 = (d11 * d20 - d01 * d21) / denom;
        w3 = (d00 * d21 - d01 * d20) / denom;
        w1 = R(1) - w2 - w3;
    } else {
        w1 = R(1);
        w2 = R(0);
        w3 = R(0);
    }
    w1 = w1 < R(0) ? R(0) : (w1 > R(1) ? R(1) : w1);
    w2 = w2 < R(0) ? R(0) : (w2 > R(1) ? R(1) : w2);
    w3 = w3 < R(0) ? R(0) : (w3 > R(1) ? R(1) : w3);
    R sum = w1 + w2 + w3;
    if (sum > R(1e-12)) {
        w1 = w1 / sum;
        w2 = w2 / sum;
        w3 = w3 / sum;
    } else {
        w1 = R(1);
        w2 = R(0);
        w3 = R(0);
    }
    V3<R> wa = xyz(S.w[ia]), wb = xyz(S.w[ib]), wc = xyz(S.w[ic]);
    pa = add(add(scale(wa, w1), scale(wb, w2)), scale(wc, w3));
    V3<R> mk = add(add(scale(va, w1), scale(vb, w2)), scale(vc, w3));
    pb = sub(pa, mk);
    normal = n;
    depth = dist;
}

// Warp-cooperative epa, epa.rs:89-189.  All lanes of the warp call it with
// the same arguments; returns true (uniformly) on convergence.  One pass over
// the faces per new vertex: faces that see it move to the visible list, the
// others close up in place, both in order.  An edge of a visible face is on
// the horizon when no other visible face has it (in either direction): the
// visible faces are counted at each vertex pair, where testing each edge
// against every visible face took most of an iteration.
// Measured per iteration of one warp: about 4,700 cycles before (hull pairs),
// bound by latency; see k_epa for whole launches.
template <class R>
__device__ bool epa_warp(EpaSmem<R>& S, const NB<R>& a, const NB<R>& b, const A4<R>* simplex, const A4<R>* hull,
                         uint32_t* err, V3<R>& normal, R& depth, V3<R>& pa, V3<R>& pb) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    if (lane < 4) {
        S.v[lane] = simplex[lane];
        S.w[lane] = simplex[4 + lane];
    }
    __syncwarp();
    uint32_t nf = 0;
    uint32_t nv = 4;
    // the lane's nearest face among those it wrote: first minimum in index order
    R near_d = R(0);
    uint32_t near_i = kAll;
    auto wrote = [&](R d, uint32_t pos) {
        if (!isnan(d) && (near_i == kAll || d < near_d)) {
            near_d = d;
            near_i = pos;
        }
    };
    {
        // the four initial faces, epa.rs:97-100, added in order
        const uint32_t init[4] = {0u | (1u << 8) | (2u << 16), 0u | (3u << 8) | (1u << 16),
                                  0u | (2u << 8) | (3u << 16), 1u | (3u << 8) | (2u << 16)};
        A4<R> nd;
        uint32_t abc;
        bool ok = false;
        if (lane < 4) ok = make_face(S, fa_(init[lane]), fb_(init[lane]), fc_(init[lane]), nd, abc);
        const uint32_t okm = __ballot_sync(kAll, ok);
        if (ok) {
            const uint32_t pos = __popc(okm & lt_mask);
            S.fnd[pos] = nd;
            S.fabc[pos] = abc;
            wrote(nd.w, pos);
        }
        nf = __popc(okm);
        __syncwarp();
    }
    for (int it = 0; it < 64; ++it) {
        // no face of nonzero area (a flat or collapsed simplex): no contact,
        // where the reference would emit its zero default face (a zero normal
        // at zero depth, whose tangents are NaN)
        if (nf == 0) return false;  // warp-uniform
        // closest face: first minimum in index order (strict <); the serial
        // scan starts from face 0, which a NaN distance there keeps
        uint32_t mi = warp_best<false>(near_i != kAll, near_d, near_i);
        if (isnan(S.fnd[0].w)) mi = 0;
        const A4<R> mnd = S.fnd[mi];
        const uint32_t mabc = S.fabc[mi];
        V3<R> sp, sw;
        support_witness_warp(a, b, xyz(mnd), hull, sp, sw, lane);
        const R sd = dot(xyz(mnd), sp);
        if (sd - mnd.w < R(1e-4)) {
            face_contact(S, mnd, mabc, normal, depth, pa, pb);
            return true;
        }
        const uint32_t ni = nv;
        if (ni >= 256u) {
            face_contact(S, mnd, mabc, normal, depth, pa, pb);
            return true;
        }
        if (lane == 0) {
            S.v[ni] = pack(sp);
            S.w[ni] = pack(sw);
        }
        nv += 1;
        // faces that see the vertex, and the others closed up
        near_i = kAll;
        uint32_t kept = 0, nvis = 0;
        for (uint32_t c = 0; c < nf; c += 32u) {
            const uint32_t i = c + lane;
            A4<R> f{};
            uint32_t abc = 0;
            bool vis = false, keep = false;
            if (i < nf) {
                f = S.fnd[i];
                abc = S.fabc[i];
                vis = dot(xyz(f), sub(sp, xyz(S.v[fa_(abc)]))) > R(0);
                keep = !vis;
            }
            const uint32_t vm = __ballot_sync(kAll, vis), km = __ballot_sync(kAll, keep);  // all have read
            if (vis) S.vis[nvis + __popc(vm & lt_mask)] = abc;
            if (keep) {
                const uint32_t pos = kept + __popc(km & lt_mask);
                S.fnd[pos] = f;
                S.fabc[pos] = abc;
                wrote(f.w, pos);
            }
            nvis += __popc(vm);
            kept += __popc(km);
            __syncwarp();
        }
        nf = kept;
        // visible faces at each of their edges
        for (uint32_t c = lane; c < nvis; c += 32u) {
            const uint32_t f = S.vis[c], x = fa_(f), y = fb_(f), z = fc_(f);
            const uint32_t e[3] = {edge_at(x, y), edge_at(y, z), edge_at(z, x)};
#pragma unroll
            for (int k = 0; k < 3; ++k) atomicAdd(&S.edge[e[k] >> 2], 1u << (8u * (e[k] & 3u)));
        }
        __syncwarp();
        // horizon: edges of one visible face, in face and edge order
        uint32_t hc = 0;
        for (uint32_t c = 0; c < nvis; c += 32u) {
            uint32_t my[3];
            uint32_t k = 0;
            if (c + lane < nvis) {
                const uint32_t f = S.vis[c + lane], v[4] = {fa_(f), fb_(f), fc_(f), fa_(f)};
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const uint32_t e = edge_at(v[q], v[q + 1]);
                    my[q] = v[q] | (v[q + 1] << 8);
                    if (((S.edge[e >> 2] >> (8u * (e & 3u))) & 0xFFu) == 1u) k |= 1u << q;
                }
            }
            // order-preserving append: one ballot per edge
            const uint32_t b0 = __ballot_sync(kAll, k & 1u), b1 = __ballot_sync(kAll, k & 2u),
                           b2 = __ballot_sync(kAll, k & 4u);
            uint32_t at = hc + __popc(b0 & lt_mask) + __popc(b1 & lt_mask) + __popc(b2 & lt_mask);
#pragma unroll
            for (int q = 0; q < 3; ++q)
                if ((k >> q) & 1u) {
                    if (at < (uint32_t)kEpaH) S.hor[at] = my[q];
                    ++at;
                }
            hc += __popc(b0) + __popc(b1) + __popc(b2);
        }
        if (hc > (uint32_t)kEpaH) {
            if (lane == 0) atomicOr(err, kErrEpaHorizon);
            hc = kEpaH;
        }
        __syncwarp();
        for (uint32_t c = lane; c < nvis; c += 32u) {
            const uint32_t f = S.vis[c], x = fa_(f), y = fb_(f), z = fc_(f);
            S.edge[edge_at(x, y) >> 2] = 0u;
            S.edge[edge_at(y, z) >> 2] = 0u;
            S.edge[edge_at(z, x) >> 2] = 0u;
        }
        // stitch the horizon to the new vertex (degenerate faces dropped)
        for (uint32_t c = 0; c < hc; c += 32u) {
            const uint32_t h = c + lane;
            A4<R> nd;
            uint32_t abc = 0;
            bool ok = false;
            if (h < hc) {
                const uint32_t e = S.hor[h];
                ok = make_face(S, ni, e & 0xFF, (e >> 8) & 0xFF, nd, abc);
            }
            const uint32_t okm = __ballot_sync(kAll, ok);
            const uint32_t pos = nf + __popc(okm & lt_mask);
            if (ok && pos < (uint32_t)kEpaF) {
                S.fnd[pos] = nd;
                S.fabc[pos] = abc;
                wrote(nd.w, pos);
            }
            const uint32_t add_n = __popc(okm);
            if (nf + add_n > (uint32_t)kEpaF) {
                if (lane == 0) atomicOr(err, kErrEpaFaces);
                nf = kEpaF;
            } else {
                nf += add_n;
            }
        }
        __syncwarp();
    }
    return false;
}

}  // namespace dio
