// k_rows.cuh -- contact rows on the device.
//
// The reference builds rows on the host each frame: AvbdSolver::raw_contact
// (engine/src/physics/gpu.rs:239-264), container_contacts (:352-404),
// finalize_contacts (:266-311: warm start by (a, b), decay, CSR).  Here each
// piece is a kernel over slots / bodies / rows:
//   k_row_counts + scans -> k_rows           rows from valid narrow slots and
//                                            container (wall / floor) rows
//   k_row_keys                               64-bit (a, b) keys + incidences
//   (radix sorts of keys / incidences)
//   k_warm                                   warm start + decay
//   k_csr_fill                               CSR idx / other-body arrays
// A world's rows are in canonical order, so k_rows warm-starts them as it
// writes them and counts the CSR's incidences on the way.
#pragma once

#include "k_narrow.cuh"

namespace dio {

// Detection-space body: pose rebased to the scene origin and rounded to R.
template <class P, class R>
__device__ __forceinline__ NB<R> load_nb(const DevWorld<P, R>& w, uint32_t i) {
    NB<R> b;
    V3<P> org{P(0), P(0), P(0)};
    if (w.origin) org = xyz(w.origin[w.scene[i]]);
    b.pos = cast3<R>(sub(xyz(w.pos[0][i]), org));
    b.rot = castq<R>(quat(w.rot[0][i]));
    b.shape = load_shape<R>(&w.shape[i]);
    return b;
}

// tangents, engine/src/physics/gpu.rs:406-414
template <class R>
__device__ __forceinline__ void tangents(V3<R> n, V3<R>& t1, V3<R>& t2) {
    V3<R> c = dabs(n.x) > R(0.9) ? cross(n, V3<R>{R(0), R(1), R(0)}) : cross(n, V3<R>{R(1), R(0), R(0)});
    t1 = normalize(c);
    t2 = cross(n, t1);
}

template <class P, class R>
__device__ __forceinline__ void write_row(const DevWorld<P, R>& w, uint32_t r, uint32_t a, uint32_t b, V3<R> n,
                                          V3<R> t1, V3<R> t2, V3<R> ra, V3<R> rb, V3<R> c0, R friction,
                                          const RowDual<P, R>& du) {
    RowStatic<R> rs;
    rs.n = pack(n, friction);
    rs.t1 = pack(t1, c0.z);
    rs.t2 = pack(t2, R(0));
    rs.ra = pack(ra, c0.x);
    rs.rb = pack(rb, c0.y);
    w.rs.put(r, rs);
    w.rd.put(r, du);
    w.ab[r] = make_uint2(a, b);
}
template <class P, class R>
__device__ __forceinline__ RowDual<P, R> fresh_dual(R kmin) {
    return RowDual<P, R>{A4<R>{kmin, kmin, kmin, R(0)}, A4<P>{P(0), P(0), P(0), P(0)}};
}
// the decay of finalize_contacts (gpu.rs:266-283)
template <class P, class R>
__device__ __forceinline__ RowDual<P, R> decay(RowDual<P, R> du, const PrepParams<R>& o) {
    P ag = P(o.alpha_gamma);
    du.lambda.x = du.lambda.x * ag;
    du.lambda.y = du.lambda.y * ag;
    du.lambda.z = du.lambda.z * ag;
    R kx = du.penalty.x * o.gamma, ky = du.penalty.y * o.gamma, kz = du.penalty.z * o.gamma;
    du.penalty.x = fmin_(fmax_(kx, o.penalty_min), o.penalty_max);
    du.penalty.y = fmin_(fmax_(ky, o.penalty_min), o.penalty_max);
    du.penalty.z = fmin_(fmax_(kz, o.penalty_min), o.penalty_max);
    return du;
}

__device__ __forceinline__ bool key_less(uint2 a, uint2 b) { return a.x < b.x || (a.x == b.x && a.y < b.y); }
__device__ __forceinline__ bool key_eq(uint2 a, uint2 b) { return a.x == b.x && a.y == b.y; }

// Where a new row's dual comes from (finalize_contacts, gpu.rs:266-283).  A
// world's rows are in canonical order: pair rows follow the pair list, which
// is sorted by (a, b), and container rows the body index, so each section is
// sorted by key with equal keys adjacent.  The first row of a key takes
// (lambda, penalty) of the last previous row with it, found from where the new
// row stands in its section (`rank`: of the key's last new row): contacts come
// and go slowly, so the search gallops out from there, and for a section that
// kept its rows it ends at once.  Every row then decays.  Without `on` (rows
// prepared for a caller) the duals start fresh and k_warm follows.
template <class P, class R>
struct WarmStart {
    bool on;
    const uint2* prev_ab;
    RowDuals<P, R> prev;
    const Counters* ctr;
    __device__ __forceinline__ RowDual<P, R> dual(uint2 key, bool first, uint32_t rank, const PrepParams<R>& o) const {
        RowDual<P, R> du = fresh_dual<P, R>(o.penalty_min);
        if (!on) return du;
        if (first) {
            const bool cont = key.y == kContainer;
            const uint32_t base = cont ? ctr->prev_pair_rows : 0u;
            uint32_t lo = base, hi = cont ? ctr->prev_rows : ctr->prev_pair_rows;
            // upper bound of key: rows before lo are at most key, rows from hi on above it
            auto above = [&](uint32_t at) { return key_less(key, prev_ab[at]); };
            if (lo < hi) {
                const uint32_t at = rank < hi - base ? base + rank : hi - 1u;
                uint32_t step = 1u;
                if (above(at)) {
                    hi = at;
                    while (lo < hi) {
                        const uint32_t g = hi - lo > step ? hi - step : lo;
                        if (!above(g)) {
                            lo = g + 1u;
                            break;
                        }
                        hi = g;
                        step <<= 1;
                    }
                } else {
                    lo = at + 1u;
                    while (lo < hi) {
                        const uint32_t g = hi - lo > step ? lo + step - 1u : hi - 1u;
                        if (above(g)) {
                            hi = g;
                            break;
                        }
                        lo = g + 1u;
                        step <<= 1;
                    }
                }
            }
            while (lo < hi) {
                const uint32_t mid = lo + ((hi - lo) >> 1);
                if (!above(mid))
                    lo = mid + 1u;
                else
                    hi = mid;
            }
            if (lo > base && key_eq(prev_ab[lo - 1], key)) {
                const RowDual<P, R> pd = prev[lo - 1];
                du.lambda = pd.lambda;
                du.penalty = pd.penalty;
            }
        }
        return decay(du, o);
    }
};

// The lanes of this lane's group of `per` slots (per divides 32) among `m`.
__device__ __forceinline__ uint32_t group_lanes(uint32_t m, uint32_t lane, uint32_t per) {
    return m & ((per == 32u ? 0xFFFFFFFFu : (1u << per) - 1u) << (lane & ~(per - 1u)));
}

// raw_contact for one valid slot, as row r; `first` of its group, which ends
// with row `last`.
template <class P, class R>
__device__ __forceinline__ void slot_row(const DevWorld<P, R>& w, const Slot<R>& s, uint32_t r, bool first,
                                         uint32_t last, const PrepParams<R>& o, const WarmStart<P, R>& warm) {
    const RowDual<P, R> du = warm.dual(make_uint2(s.a, s.b), first, last, o);
    const NB<R> A = load_nb(w, s.a), B = load_nb(w, s.b);
    V3<R> nrm = xyz(s.normal);
    V3<R> t1, t2;
    tangents(nrm, t1, t2);
    V3<R> ra = rotate(conj(A.rot), sub(xyz(s.pa), A.pos));
    V3<R> rb = rotate(conj(B.rot), sub(xyz(s.pb), B.pos));
    write_row(w, r, s.a, s.b, neg(nrm), t1, t2, ra, rb, V3<R>{o.margin - s.depth, R(0), R(0)}, o.friction, du);
}

// cube_support_face, engine/src/physics/gpu.rs:314-350 (per-axis for BOX)
template <class R>
__device__ __forceinline__ void support_face(const NB<R>& b, V3<R> outward, V3<R> pts[4]) {
    V3<R> ax[3];
    axes_of(b.rot, ax);
    uint32_t ai = 0;
    R best = dabs(dot(ax[0], outward));
    for (uint32_t i = 1; i < 3; ++i) {
        R al = dabs(dot(ax[i], outward));
        if (al > best) {
            ai = i;
            best = al;
        }
    }
    V3<R> h = box_half(b.shape);
    V3<R> center, u, v;
    R eu, ev;
    face_frame(b.pos, ax, h, ai, outward, pts, center, u, v, eu, ev);
}

// container_contacts for one body (engine/src/physics/gpu.rs:352-404):
// counts (write == false) or writes rows starting at `r`; `last`: its last
// row's place among the container rows.
template <class P, class R>
__device__ __forceinline__ uint32_t container_rows(const DevWorld<P, R>& w, uint32_t i, const PrepParams<R>& o,
                                                   bool write_out, uint32_t r, uint32_t last,
                                                   const WarmStart<P, R>& warm) {
    const A4<R>* walls = w.walls + 6 * (size_t)w.scene[i];
    V3<R> vel = cast3<R>(xyz(w.vel[i]));
    // Quick reject: every support point lies within an L1 bounding radius of
    // the body centre, so when the centre plus that radius plus this step's
    // travel is (with rounding slack) inside a wall, that wall has no row
    // with depth > 0 -- the same empty set the full test produces.  The
    // bound needs only the shape's tag and first corner and the position, so
    // the orientation and the rest of the shape are read only for a body
    // that can reach a wall.
    const uint32_t tag = reinterpret_cast<const uint4*>(&w.shape[i])->x;
    const float4 c0 = reinterpret_cast<const float4*>(w.shape[i].corners)[0];
    V3<P> org{P(0), P(0), P(0)};
    if (w.origin) org = xyz(w.origin[w.scene[i]]);
    const V3<R> pos = cast3<R>(sub(xyz(w.pos[0][i]), org));  // as load_nb forms it
    const bool boxy = tag == DIO_SHAPE_CUBE || tag == DIO_SHAPE_BOX;
    R rbound = R(-1);
    const bool hull = tag == DIO_SHAPE_HULL && w.hull_bound;
    if (hull) {
        // over its vertices, kept from the upload; an orientation that is not
        // of unit length scales them by its square
        const Q4<R> q = narrowq<R>(quat(w.rot[0][i]));
        rbound = w.hull_bound[i] * fmax_(R(1), q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
    } else if (boxy) {
        rbound = dabs(R(c0.x)) + dabs(R(c0.y)) + dabs(R(c0.z));
    } else if (tag == DIO_SHAPE_SPHERE) {
        rbound = dabs(R(c0.x));
    } else if (tag == DIO_SHAPE_TETRAHEDRON) {
        const ShapeR<R> sh = load_shape<R>(&w.shape[i]);
        rbound = R(0);
        for (int k = 0; k < 4; ++k)
            rbound = fmax_(rbound, dabs(sh.c[k].x) + dabs(sh.c[k].y) + dabs(sh.c[k].z));
    }
    const R travel = rbound >= R(0) ? length(vel) * o.dt : R(0);
    uint32_t reach = 0x3Fu;  // walls a support point may reach this step
    if (rbound >= R(0)) {
        reach = 0;
        for (int k = 0; k < 6; ++k) {
            const A4<R> wall = walls[k];
            const R d = dot(pos, xyz(wall));
            R far = rbound + travel, mag = dabs(d);
            if (hull) {
                // a vertex may lie on its bound: the wall's normal is taken with
                // its length (a container's rotation need not be a unit one), and
                // the rounding of d with its terms
                far = far * (R(1.0001) * fmax_(R(1), dot(xyz(wall), xyz(wall))));
                mag = dabs(pos.x * wall.x) + dabs(pos.y * wall.y) + dabs(pos.z * wall.z);
            }
            const R slack = R(1e-4) * (R(1) + dabs(wall.w) + mag);
            if (!(d + far + slack < wall.w)) reach |= 1u << k;
        }
    }
    if (!reach) return 0;
    NB<R> b = load_nb(w, i);
    uint32_t count = 0;
#pragma unroll 1
    for (int k = 0; k < 6; ++k) {
        if (!((reach >> k) & 1u)) continue;
        const A4<R> wall = walls[k];
        const V3<R> outward = xyz(wall);
        const R plane = wall.w;
        V3<R> pts[4];
        uint32_t np;
        if (boxy) {
            support_face(b, outward, pts);
            np = 4;
        } else {
            V3<R> local = rotate(conj(b.rot), outward);
            pts[0] = add(rotate(b.rot, support(b.shape, local, w.hull)), b.pos);
            np = 1;
        }
        V3<R> normal = neg(outward);
        V3<R> t1, t2;
        if (write_out) tangents(normal, t1, t2);
        for (uint32_t p = 0; p < np; ++p) {
            V3<R> cp = pts[p];
            R cur = dot(cp, outward) - plane;
            V3<R> pred = add(cp, scale(vel, o.dt));
            R pd = dot(pred, outward) - plane;
            R depth = fmax_(cur, pd);
            if (depth > R(0)) {
                if (write_out) {
                    if (r + count < w.max_rows) {
                        V3<R> ra = rotate(conj(b.rot), sub(cp, b.pos));
                        write_row(w, r + count, i, kContainer, normal, t1, t2, ra, V3<R>{R(0), R(0), R(0)},
                                  V3<R>{o.margin - depth, R(0), R(0)}, o.friction,
                                  warm.dual(make_uint2(i, kContainer), count == 0, last, o));
                    } else {
                        atomicOr(&w.ctr->error_flags, kErrRowOverflow);
                    }
                }
                ++count;
            }
        }
    }
    return count;
}

// An L1 bounding radius of each hull body's vertices (a little over, for the
// rounding of their rotation), once per upload.
template <class P, class R>
__global__ void k_hull_bounds(DevWorld<P, R> w, uint32_t n, R* bound) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint4 h = *reinterpret_cast<const uint4*>(&w.shape[i]);
        if (h.x != DIO_SHAPE_HULL) continue;
        R b = R(0);
        bool finite = true;
        for (uint32_t k = 0; k < h.z; ++k) {
            const V3<R> v = xyz(w.hull[h.y + k]);
            const R l = dabs(v.x) + dabs(v.y) + dabs(v.z);
            finite = finite && finite_(l);
            b = fmax_(b, l);
        }
        bound[i] = finite ? b * R(1.0001) : R(-1);  // -1: no bound, the full test
    }
}

// Wall k of a scene's container (container_collide,
// engine/src/physics/gpu.rs): outward normal = rotation * (+-axis), plane
// offset = centre . outward + half extent; centre rebased to the scene's
// detection origin.
template <class P, class R>
__device__ __forceinline__ A4<R> scene_wall(const SceneDesc& sc, V3<P> org, uint32_t k) {
    const V3<R> center = cast3<R>(sub(V3<P>{P(sc.center[0]), P(sc.center[1]), P(sc.center[2])}, org));
    const Q4<R> crot{R(sc.rotation[0]), R(sc.rotation[1]), R(sc.rotation[2]), R(sc.rotation[3])};
    const R half = R(sc.half_extent);
    const V3<R> axis = k < 2 ? V3<R>{R(1), R(0), R(0)} : (k < 4 ? V3<R>{R(0), R(1), R(0)} : V3<R>{R(0), R(0), R(1)});
    const R sign = (k & 1) ? R(-1) : R(1);
    const V3<R> outward = rotate(crot, scale(axis, sign));
    return A4<R>{outward.x, outward.y, outward.z, dot(center, outward) + half};
}
// every scene's walls, once per upload
template <class P, class R>
__global__ void k_scene_walls(DevWorld<P, R> w, const SceneDesc* scenes, uint32_t ns, A4<R>* walls) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < 6 * ns; t += gridDim.x * blockDim.x) {
        const uint32_t s = t / 6, k = t % 6;
        V3<P> org{P(0), P(0), P(0)};
        if (w.origin) org = xyz(w.origin[s]);
        walls[t] = scene_wall<P, R>(scenes[s], org, k);
    }
}
// The scene table of a caller's single scene: given by value, so that the host
// waits for no copy (chunk: it is one of the shared-memory trees).
template <class P, class R>
__global__ void k_single_scene(const SceneDesc sc, bool chunk, SceneDesc* scenes, uint2* chunks, A4<R>* walls) {
    const uint32_t k = threadIdx.x;
    if (k < 6u) walls[k] = scene_wall<P, R>(sc, V3<P>{P(0), P(0), P(0)}, k);
    if (k == 0u) {
        scenes[0] = sc;
        if (chunk) chunks[0] = make_uint2(0u, 1u);
    }
}

// Valid slots of each live group of `per` slots (the first min(*ng_dev, ng)
// groups) and container rows of each of the bodies [0, n); counts2[n] is set
// to 0 for the exclusive scan over n + 1 entries, and so is incident[0 .. n]
// (if given).
template <class P, class R>
__global__ void k_row_counts(DevWorld<P, R> w, const Slot<R>* slots, uint32_t per, const uint32_t* ng_dev, uint32_t ng,
                             uint32_t n, PrepParams<R> o, uint32_t* counts, uint32_t* counts2, uint32_t* incident) {
    pdl_enter();
    if (ng_dev) ng = min(*ng_dev, ng);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        counts2[n] = 0u;
        if (incident) incident[n] = 0u;
    }
    const WarmStart<P, R> none{};
    // bodies first (up to a warp's multiple, so that a group's slots are one
    // warp's): they are known to be there, and the longer work
    const uint32_t nw = (n + 31u) & ~31u, lane = threadIdx.x & 31u;
    const uint64_t items = (uint64_t)nw + (uint64_t)ng * per;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t - lane < items;
         t += (uint64_t)gridDim.x * blockDim.x) {
        if (t < nw) {
            const uint32_t i = (uint32_t)t;
            if (i >= n) continue;
            uint32_t c = 0;
            if (w.inv[i].w != R(0) && w.scenes[w.scene[i]].has_container) c = container_rows(w, i, o, false, 0, 0, none);
            counts2[i] = c;
            if (incident) incident[i] = 0u;
        } else {
            const uint64_t k = t - nw;
            const uint32_t valid = __ballot_sync(0xFFFFFFFFu, t < items && slots[k].valid);
            if (t < items && (lane & (per - 1u)) == 0u)
                counts[k / per] = (uint32_t)__popc(group_lanes(valid, lane, per));
        }
    }
}

// The rows: pair rows at off[group] (total at off[ng], the capacity), then
// container rows at off2[body].  incident (may be null, zero on entry): the
// dynamic-body CSR's counters, each body's rows counted.
template <class P, class R>
__global__ void k_rows(DevWorld<P, R> w, const Slot<R>* slots, uint32_t per, const uint32_t* ng_dev, uint32_t ng,
                       uint32_t n, PrepParams<R> o, const uint32_t* off, const uint32_t* off2, WarmStart<P, R> warm,
                       uint32_t* incident) {
    pdl_enter();
    const uint32_t live = ng_dev ? min(*ng_dev, ng) : ng;
    const uint32_t pair_rows = off[ng], cont_rows = off2[n];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // rows that are kept: the next step's warm start searches that many
        w.ctr->pair_rows = min(pair_rows, w.max_rows);
        w.ctr->container_rows = cont_rows;
        const uint64_t t = (uint64_t)pair_rows + cont_rows;
        w.ctr->rows = t > w.max_rows ? w.max_rows : (uint32_t)t;
        if (t > w.max_rows) atomicOr(&w.ctr->error_flags, kErrRowOverflow);
    }
    // a thread a slot: the rows of a contact-dense pair are written together
    // (a thread a group wrote up to eight in turn: 20 us cold for 90 pairs of
    // cubes, now 8; 200,000-body wall 94 and 74, with the galloping warm start)
    const uint64_t nslots = (uint64_t)live * per, sw = (nslots + 31u) & ~31ull, items = sw + n;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t - lane < items;
         t += (uint64_t)gridDim.x * blockDim.x) {
        if (t < sw) {
            const uint32_t p = (uint32_t)(t / per);
            uint32_t r = 0;
            bool good = false;
            Slot<R> s;
            // a group without valid slots (a box overlap without contact) is
            // skipped unread; the last live group ends at the total
            if (t < nslots && (p + 1 < live ? off[p + 1] : pair_rows) != (r = off[p])) {
                s = slots[t];
                good = s.valid;
                if (good && (s.a >= w.n || s.b >= w.n)) {
                    atomicOr(&w.ctr->error_flags, kErrBadIndex);
                    good = false;
                }
            }
            const uint32_t rows = group_lanes(__ballot_sync(0xFFFFFFFFu, good), lane, per);
            r += (uint32_t)__popc(rows & ((1u << lane) - 1u));
            if (good && r >= w.max_rows) {
                atomicOr(&w.ctr->error_flags, kErrRowOverflow);
                good = false;
            }
            const uint32_t kept = group_lanes(__ballot_sync(0xFFFFFFFFu, good), lane, per);
            if (!good) continue;
            const bool first = !(kept & ((1u << lane) - 1u));
            if (incident && first) {  // a group's slots are one pair's
                if (w.inv[s.a].w != R(0)) atomicAdd(&incident[s.a], (uint32_t)__popc(kept));
                if (w.inv[s.b].w != R(0)) atomicAdd(&incident[s.b], (uint32_t)__popc(kept));
            }
            slot_row(w, s, r, first, r + (uint32_t)__popc(kept) - 1u, o, warm);
        } else {
            const uint64_t b = t - sw;
            if (b >= n) continue;
            const uint32_t i = (uint32_t)b, r = off2[i], rows = off2[i + 1] - r;
            if (!rows) continue;  // nothing to recompute
            container_rows(w, i, o, true, pair_rows + r, r + rows - 1u, warm);
            if (incident) {  // rows that were kept
                const uint64_t at = (uint64_t)pair_rows + r;
                const uint32_t kept = at >= w.max_rows ? 0u : (uint32_t)min((uint64_t)rows, w.max_rows - at);
                if (kept) atomicAdd(&incident[i], kept);
            }
        }
    }
}

__device__ __forceinline__ unsigned long long row_key(uint2 ab) {
    return ((unsigned long long)ab.x << 32) | (unsigned long long)ab.y;
}

// Keys + row ids for the warm-start sorts, and the (body, row) incidences of
// the CSR (two per row; b == CONTAINER becomes the sentinel body `n`).
static __global__ void k_row_keys(const uint2* ab, const uint32_t* m_dev, uint32_t cap, unsigned long long* keys,
                           uint32_t* ids, uint32_t* inc_body, uint32_t* inc_row, uint32_t n_sentinel) {
    uint32_t m = *m_dev;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < cap; r += gridDim.x * blockDim.x) {
        if (r < m) {
            uint2 v = ab[r];
            if (keys) {
                keys[r] = row_key(v);
                ids[r] = r;
            }
            if (inc_body) {
                inc_body[2 * r] = v.x;
                inc_row[2 * r] = r;
                inc_body[2 * r + 1] = v.y == kContainer ? n_sentinel : v.y;
                inc_row[2 * r + 1] = r;
            }
        } else {
            if (keys) {
                keys[r] = ~0ull;
                ids[r] = r;
            }
            if (inc_body) {
                inc_body[2 * r] = n_sentinel;
                inc_row[2 * r] = r;
                inc_body[2 * r + 1] = n_sentinel;
                inc_row[2 * r + 1] = r;
            }
        }
    }
}

// Warm start + decay (finalize_contacts, gpu.rs:266-283).  new_keys/new_ids
// are the new rows' keys stably sorted; prev_keys/prev_ids the previous
// rows'.  The first new row of each key takes (lambda, penalty) of the LAST
// previous row with that key; every row then decays.
template <class P, class R>
__global__ void k_warm(DevWorld<P, R> w, const uint32_t* m_dev, const unsigned long long* new_keys,
                       const uint32_t* new_ids, const unsigned long long* prev_keys, const uint32_t* prev_ids,
                       uint32_t n_prev, RowDuals<P, R> prev_dual, PrepParams<R> o) {
    uint32_t m = *m_dev;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < m; t += gridDim.x * blockDim.x) {
        unsigned long long key = new_keys[t];
        uint32_t r = new_ids[t];
        RowDual<P, R> du = w.rd[r];
        bool first = t == 0 || new_keys[t - 1] != key;
        if (first && n_prev > 0) {
            // upper bound of key in prev_keys -> last occurrence is ub - 1
            uint32_t lo = 0, hi = n_prev;
            while (lo < hi) {
                uint32_t mid = (lo + hi) >> 1;
                if (prev_keys[mid] <= key)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            if (lo > 0 && prev_keys[lo - 1] == key) {
                const RowDual<P, R> pd = prev_dual[prev_ids[lo - 1]];
                du.lambda = pd.lambda;
                du.penalty = pd.penalty;
            }
        }
        w.rd.put(r, decay(du, o));
    }
}

// Per-body counts of the sorted incidences -> offsets are the exclusive
// scan; the fill keeps the sorted (row-ascending) order per body.
static __global__ void k_inc_count(const uint32_t* inc_body_sorted, const uint32_t* m_dev, uint32_t n, uint32_t* counts) {
    uint32_t total = 2 * *m_dev;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < total; j += gridDim.x * blockDim.x) {
        uint32_t b = inc_body_sorted[j];
        if (b < n) atomicAdd(&counts[b], 1u);
    }
}

template <class P, class R>
__global__ void k_csr_fill(DevWorld<P, R> w, const uint32_t* inc_body_sorted, const uint32_t* inc_row_sorted,
                           const uint32_t* m_dev) {
    uint32_t total = 2 * *m_dev;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < total; j += gridDim.x * blockDim.x) {
        uint32_t b = inc_body_sorted[j];
        if (b >= w.n) continue;  // container sentinels sort last
        uint32_t r = inc_row_sorted[j];
        uint2 ab = w.ab[r];
        uint32_t oth;
        if (ab.y == kContainer)
            oth = kContainer;
        else if (ab.x == b)
            oth = ab.y;
        else
            oth = ab.x | kIsB;
        if (j < w.max_incid) {
            w.row_idx[j] = r;
            w.row_oth[j] = oth;
        }
    }
}

// ---- device-driven variants for the resident world (no host-known counts)

// roll the per-step counters: the finished step's row counts become the
// warm-start source, the per-step counts restart at zero (and up to two
// scratch words the step's scans and sorts expect zeroed, if given)
static __global__ void k_roll_counters(Counters* c, uint32_t* zero0, uint32_t* zero1) {
    if (zero0) *zero0 = 0u;
    if (zero1) *zero1 = 0u;
    c->prev_rows = c->rows;
    c->prev_pair_rows = c->pair_rows;
    c->prev_pairs = c->pairs;
    c->pairs = 0;
    c->rows = 0;
    c->pair_rows = 0;
    c->container_rows = 0;
    c->gjk_work = 0;
    c->epa_work = 0;
    c->epa_next = 0;
    c->colors = 0;
    c->traverse_pairs = 0;
    c->failed_solves = 0;
}

// CSR of the dynamic bodies only (the primal never visits a static body):
// counts from k_rows, an atomic scatter (each body's count taken down to
// zero) into `loose`, then each row's place in its body's segment by its rank
// there, which restores the reference's fill order (finalize_contacts,
// gpu.rs:286-310) without a sort over all incidences, with the other-body
// array.
// remaining: each body's incidence count (k_rows), consumed here
template <class P, class R>
__global__ void k_csr_scatter_dyn(DevWorld<P, R> w, uint32_t* remaining, uint32_t* loose) {
    pdl_enter();
    const uint32_t m = w.ctr->rows;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < m; r += gridDim.x * blockDim.x) {
        uint2 ab = w.ab[r];
        if (w.inv[ab.x].w != R(0)) {
            uint32_t j = w.row_off[ab.x] + atomicSub(&remaining[ab.x], 1u) - 1u;
            if (j < w.max_incid) loose[j] = r;
        }
        if (ab.y != kContainer && w.inv[ab.y].w != R(0)) {
            uint32_t j = w.row_off[ab.y] + atomicSub(&remaining[ab.y], 1u) - 1u;
            if (j < w.max_incid) loose[j] = r;
        }
    }
}

// A thread per end of a row counts the smaller rows of its body's segment: the
// loads do not wait for one another, and the threads of a pair's rows read the
// same ones.  (A thread per body with an insertion sort in local memory, longer
// segments by a CTA each: 15 us cold a step for 8,192 stacked cubes, 13.5 for a
// 55-cube pyramid of 8-contact pairs; now 6 and 5.)  Counting needs no buffer,
// so a segment may have any length: every entry that the solve walks is written.
// (A plate of 3,455 and of 9,705 rows: the whole rows phase 106 and 290 us a
// step, beside a solve of 2,200 and 6,600 for that body's sums.)
template <class P, class R>
__global__ void k_csr_finish_dyn(DevWorld<P, R> w, const uint32_t* loose) {
    pdl_enter();
    const uint64_t items = 2ull * w.ctr->rows;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < items; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(t >> 1);
        const uint2 ab = w.ab[r];
        const uint32_t i = (t & 1u) ? ab.y : ab.x;
        if (i == kContainer || w.inv[i].w == R(0)) continue;
        const uint32_t j0 = w.row_off[i], j1 = min(w.row_off[i + 1], w.max_incid);
        uint32_t j = j0;
#pragma unroll 8
        for (uint32_t q = j0; q < j1; ++q) j += loose[q] < r ? 1u : 0u;
        if (j >= j1) continue;
        w.row_idx[j] = r;
        w.row_oth[j] = ab.y == kContainer ? kContainer : ((t & 1u) ? (ab.x | kIsB) : ab.y);
    }
}

}  // namespace dio
