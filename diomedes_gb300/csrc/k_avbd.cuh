// k_avbd.cuh -- AVBD init / primal / dual / recover on sm_103a.
//
// Restates engine/gpu_physics/avbd/src/lib.rs:202-699.  Differences in
// structure (not in arithmetic):
//   * SoA poses (16-byte vector loads) instead of AoS Vec4 buffers.
//   * Contacts are read through a per-body CSR that also carries the other
//     body and the a/b side, so the row's (a, b) never has to be fetched.
//   * Joints are read through a per-body joint CSR in joint order instead of
//     the reference's scan over every joint for every body (O(N J)); the
//     accumulation order per body is unchanged.
//   * P (pose precision) may be double: inertial targets, poses and lambda
//     accumulate in FP64 while the 6x6 Hessian, LDL^T and rows stay in R.
//   * The final pose is also left in buffer 0, so a device-resident world
//     starts every step from buffer 0.
#pragma once

#include <type_traits>

#include "div_rn.cuh"
#include "engine.cuh"

namespace dio {

template <class R>
struct Block6 {
    R h[21];  // lower triangle, row-major: (0,0) (1,0) (1,1) (2,0) ...
    R g[6];
};

__device__ __forceinline__ constexpr int tri(int i, int j) { return i * (i + 1) / 2 + j; }

// H += J J^T k, g += J f (add_constraint_row, avbd/src/lib.rs:182-198)
template <class R>
__device__ __forceinline__ void stamp(Block6<R>& B, V3<R> jl, V3<R> ja, R k, R f) {
    const R J[6] = {jl.x, jl.y, jl.z, ja.x, ja.y, ja.z};
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) B.h[tri(i, j)] = B.h[tri(i, j)] + J[i] * J[j] * k;
#pragma unroll
    for (int i = 0; i < 6; ++i) B.g[i] = B.g[i] + J[i] * f;
}

// stamp() for a row whose Jacobian entries outside MASK are exact zeros
// (a ball-socket axis row: J = (s e_k, r x s e_k)).  The H terms with a zero
// factor are +-0 when J and k are finite, and adding +-0 leaves an H entry
// unchanged because a round-to-nearest sum that starts at +0 (or at the
// positive diagonal) is never -0; so skipping them is exact.  g takes all
// six terms (its start values can be -0).  Callers check finiteness first.
template <int MASK, class R>
__device__ __forceinline__ void stamp_masked(Block6<R>& B, V3<R> jl, V3<R> ja, R k, R f) {
    const R J[6] = {jl.x, jl.y, jl.z, ja.x, ja.y, ja.z};
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j)
            if (((MASK >> i) & 1) && ((MASK >> j) & 1)) B.h[tri(i, j)] = B.h[tri(i, j)] + J[i] * J[j] * k;
#pragma unroll
    for (int i = 0; i < 6; ++i) B.g[i] = B.g[i] + J[i] * f;
}
constexpr int kMaskAxisX = (1 << 0) | (1 << 4) | (1 << 5);  // J = (s, 0, 0, 0, s r.z, -s r.y)
constexpr int kMaskAxisY = (1 << 1) | (1 << 3) | (1 << 5);  // J = (0, s, 0, -s r.z, 0, s r.x)
constexpr int kMaskAxisZ = (1 << 2) | (1 << 3) | (1 << 4);  // J = (0, 0, s, s r.y, -s r.x, 0)

// solve6, avbd/src/lib.rs:107-180 (unpivoted LDL^T); solves H x = -g.
// div(p, v): a column's quotients by pivot p in place; div.each(p, v): one by
// each pivot.
template <class R, class Div>
__device__ __forceinline__ void solve6_with(const Block6<R>& B, R x[6], Div&& div) {
    const R* H = B.h;
    R a11 = H[tri(0, 0)], a21 = H[tri(1, 0)], a31 = H[tri(2, 0)], a22 = H[tri(1, 1)], a32 = H[tri(2, 1)],
      a33 = H[tri(2, 2)];
    R a41 = H[tri(3, 0)], a51 = H[tri(4, 0)], a61 = H[tri(5, 0)], a42 = H[tri(3, 1)], a52 = H[tri(4, 1)],
      a62 = H[tri(5, 1)];
    R a43 = H[tri(3, 2)], a53 = H[tri(4, 2)], a63 = H[tri(5, 2)];
    R a44 = H[tri(3, 3)], a54 = H[tri(4, 3)], a64 = H[tri(5, 3)], a55 = H[tri(4, 4)], a65 = H[tri(5, 4)],
      a66 = H[tri(5, 5)];
    const Pivot<R> p1 = div.pivot(a11);
    R c1[5] = {a21, a31, a41, a51, a61};
    div(p1, c1);
    R l21 = c1[0], l31 = c1[1], l41 = c1[2], l51 = c1[3], l61 = c1[4];
    R d1 = a11;
    R d2 = a22 - l21 * l21 * d1;
    const Pivot<R> p2 = div.pivot(d2);
    R c2[4] = {a32 - l21 * l31 * d1, a42 - l21 * l41 * d1, a52 - l21 * l51 * d1, a62 - l21 * l61 * d1};
    div(p2, c2);
    R l32 = c2[0], l42 = c2[1], l52 = c2[2], l62 = c2[3];
    R d3 = a33 - (l31 * l31 * d1 + l32 * l32 * d2);
    const Pivot<R> p3 = div.pivot(d3);
    R c3[3] = {a43 - l31 * l41 * d1 - l32 * l42 * d2, a53 - l31 * l51 * d1 - l32 * l52 * d2,
               a63 - l31 * l61 * d1 - l32 * l62 * d2};
    div(p3, c3);
    R l43 = c3[0], l53 = c3[1], l63 = c3[2];
    R d4 = a44 - (l41 * l41 * d1 + l42 * l42 * d2 + l43 * l43 * d3);
    const Pivot<R> p4 = div.pivot(d4);
    R c4[2] = {a54 - l41 * l51 * d1 - l42 * l52 * d2 - l43 * l53 * d3,
               a64 - l41 * l61 * d1 - l42 * l62 * d2 - l43 * l63 * d3};
    div(p4, c4);
    R l54 = c4[0], l64 = c4[1];
    R d5 = a55 - (l51 * l51 * d1 + l52 * l52 * d2 + l53 * l53 * d3 + l54 * l54 * d4);
    const Pivot<R> p5 = div.pivot(d5);
    R c5[1] = {a65 - l51 * l61 * d1 - l52 * l62 * d2 - l53 * l63 * d3 - l54 * l64 * d4};
    div(p5, c5);
    R l65 = c5[0];
    R d6 = a66 - (l61 * l61 * d1 + l62 * l62 * d2 + l63 * l63 * d3 + l64 * l64 * d4 + l65 * l65 * d5);
    const Pivot<R> p[6] = {p1, p2, p3, p4, p5, div.pivot(d6)};
    R b0 = -B.g[0], b1 = -B.g[1], b2 = -B.g[2], b3 = -B.g[3], b4 = -B.g[4], b5 = -B.g[5];
    R z[6];
    z[0] = b0;
    z[1] = b1 - l21 * z[0];
    z[2] = b2 - l31 * z[0] - l32 * z[1];
    z[3] = b3 - l41 * z[0] - l42 * z[1] - l43 * z[2];
    z[4] = b4 - l51 * z[0] - l52 * z[1] - l53 * z[2] - l54 * z[3];
    z[5] = b5 - l61 * z[0] - l62 * z[1] - l63 * z[2] - l64 * z[3] - l65 * z[4];
    div.each(p, z);
    x[5] = z[5];
    x[4] = z[4] - l65 * x[5];
    x[3] = z[3] - l54 * x[4] - l64 * x[5];
    x[2] = z[2] - l43 * x[3] - l53 * x[4] - l63 * x[5];
    x[1] = z[1] - l32 * x[2] - l42 * x[3] - l52 * x[4] - l62 * x[5];
    x[0] = z[0] - l21 * x[1] - l31 * x[2] - l41 * x[3] - l51 * x[4] - l61 * x[5];
}

// Each quotient by a pivot is the IEEE quotient: one reciprocal per pivot and
// a correction step per quotient (div_rn.cuh), with one range test for the
// whole system (OneTest) or one per column, whose quotients are formed again
// when it fails (ColumnTests).
template <class R>
struct OneTest {
    Quotients<R> q;
    bool ok = true;
    __device__ __forceinline__ Pivot<R> pivot(R b) {
        const Pivot<R> p(b);
        ok = ok && p.ok();
        return p;
    }
    template <int N>
    __device__ __forceinline__ void operator()(const Pivot<R>& p, R (&v)[N]) {
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = q.div(p, v[k]);
    }
    __device__ __forceinline__ void each(const Pivot<R> (&p)[6], R (&v)[6]) {
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k] = q.div(p[k], v[k]);
    }
};
template <class R>
struct ColumnTests {
    __device__ __forceinline__ Pivot<R> pivot(R b) const { return Pivot<R>(b); }
    template <int N>
    __device__ __forceinline__ void operator()(const Pivot<R>& p, R (&v)[N]) const {
        divide_all(p, v);
    }
    __device__ __forceinline__ void each(const Pivot<R> (&p)[6], R (&v)[6]) const { divide_each(p, v); }
};
// hint: where a caller remembers that its systems have failed the one test.
// Such systems come again in every iteration, and a warp that solves one twice
// holds up its colour or phase (us a step or launch, all quotients divided
// again, then as it is: 13 coloured scenes without such a body 178, with one 236
// and 199; 33 scenes 113 and 98; the 400 x 500 split wall, where four systems in
// five fail, 106 and 101).  The second solve is in line: through a call, the
// system goes to local memory on every solve, and 1024 scenes take 2816 us a
// pass instead of 2610; with a test per column alone 2658.
struct NoHint {
    __device__ __forceinline__ bool careful() const { return false; }
    __device__ __forceinline__ void be_careful() const {}
};
template <class R, class Hint = NoHint>
__device__ __forceinline__ void solve6(const Block6<R>& B, R x[6], const Hint& hint = Hint()) {
    bool done = false;
    if constexpr (sizeof(R) == 4) {
        if (!hint.careful()) {
            OneTest<R> div;
            solve6_with(B, x, div);
            done = div.ok && div.q.in_range();
            if (!done) hint.be_careful();
        }
    }
    if (!done) solve6_with(B, x, ColumnTests<R>());
}

// avbd_init, avbd/src/lib.rs:202-254, for one body: the inertial target and
// the diagonal m / dt^2, I / dt^2 go to index `at` of their arrays, the
// step-start pose and the (for dynamic bodies) warm-started one come back.
template <class P>
struct InitPose {
    A4<P> start_pos, start_rot, pos, rot;
};
template <class P, class R>
__device__ __forceinline__ InitPose<P> init_pose(const DevWorld<P, R>& w, uint32_t i, uint32_t at,
                                                 const SolveParams<R>& o) {
    InitPose<P> r;
    r.pos = w.pos[0][i];
    r.rot = w.rot[0][i];
    const A4<R> inv = w.inv[i];
    const R inv_mass = inv.w;
    V3<P> pos = xyz(r.pos);
    Q4<P> rot = quat(r.rot);
    V3<P> vel = xyz(w.vel[i]);
    V3<P> ang = xyz(w.ang[i]);
    P dt = P(o.dt);
    V3<P> g{P(o.gx), P(o.gy), P(o.gz)};
    r.start_pos = pack(pos);
    r.start_rot = r.rot;
    V3<P> ip = add(pos, scale(vel, dt));
    if (inv_mass > R(0)) ip = add(ip, scale(g, dt * dt));
    w.inert_pos[at] = pack(ip);
    Q4<P> irot = quat_step(rot, scale(ang, dt));
    w.inert_rot[at] = packq(narrowq<R>(irot));
    if (w.mdt2 && inv_mass != R(0)) {
        // the primal's diagonal, constant over the step (avbd/src/lib.rs:293-296)
        const R mass = R(1) / inv.w;
        const V3<R> moment{R(1) / inv.x, R(1) / inv.y, R(1) / inv.z};
        const R dt2 = o.dt * o.dt;
        const V3<R> idt2 = divs(moment, dt2);
        w.mdt2[at] = A4<R>{mass / dt2, idt2.x, idt2.y, idt2.z};
    }
    if (inv_mass > R(0)) {
        // adaptive gravity weight, clamped to [0, 1]: formed in R in the split
        // mode (it only scales the warm-start offset)
        using Fq = std::conditional_t<std::is_same<P, R>::value, P, R>;
        const Fq dtf = Fq(o.dt);
        const V3<Fq> gf{Fq(o.gx), Fq(o.gy), Fq(o.gz)};
        V3<Fq> accel = divs(cast3<Fq>(sub(vel, xyz(w.prev_vel[i]))), dtf);
        Fq gm = length(gf);
        Fq wgt = Fq(0);
        if (gm > Fq(0)) {
            wgt = dot(accel, divs(gf, gm)) / gm;
            wgt = wgt < Fq(0) ? Fq(0) : (wgt > Fq(1) ? Fq(1) : wgt);
        }
        r.pos = pack(add(add(pos, scale(vel, dt)), scale(g, P(wgt) * dt * dt)));
        r.rot = packq(irot);  // the same quat_step(rot, ang dt)
    }
    return r;
}

// What the rows of a body take from it: its rotation rounded to R and its
// displacement since the step start, linear and angular, formed once per pose
// (each row and dual formed them again from four pose records a body).
template <class R>
struct Moved {
    V3<R> dl, da;
    Q4<R> q;
};
template <class R, class P>
__device__ __forceinline__ Moved<R> moved_from(A4<P> pos, Q4<R> q, A4<P> start_pos, A4<P> start_rot) {
    Moved<R> m;
    m.dl = narrow3<R>(sub(xyz(pos), xyz(start_pos)));
    m.q = q;
    m.da = ang_diff(q, narrowq<R>(quat(start_rot)));
    return m;
}
template <class P, class R>
__device__ __forceinline__ void put_moved(const DevWorld<P, R>& w, int buf, uint32_t i, const Moved<R>& m) {
    if constexpr (sizeof(P) != sizeof(R)) w.rot_r[buf][i] = packq(m.q);
    w.moved_l[buf][i] = pack(m.dl, m.da.x);
    w.moved_a[buf][i] = V2<R>{m.da.y, m.da.z};
}
template <class R>
__device__ __forceinline__ Moved<R> moved_of(A4<R> q, A4<R> l, V2<R> a) {
    return Moved<R>{xyz(l), V3<R>{l.w, a.x, a.y}, quat(q)};
}

// avbd_init with the poses in global memory (+ seeding buffer 1 with the
// un-warm-started pose, render/gpu_physics.rs:479-482)
template <class P, class R>
__device__ __forceinline__ void init_body(const DevWorld<P, R>& w, uint32_t i, const SolveParams<R>& o) {
    const A4<P> p4 = w.pos[0][i];
    const InitPose<P> r = init_pose(w, i, i, o);
    const R inv_mass = w.inv[i].w;
    // buffer 1 holds the un-warm-started pose for bodies the primal never
    // writes (static ones); a dynamic body's copy is overwritten by the first
    // primal before anything reads it, unless there is no iteration at all
    if (inv_mass == R(0) || o.iterations == 0) {
        w.pos[1][i] = p4;
        w.rot[1][i] = r.start_rot;
    }
    w.init_pos[i] = r.start_pos;
    w.init_rot[i] = r.start_rot;
    if (inv_mass > R(0)) {
        w.pos[0][i] = r.pos;
        w.rot[0][i] = r.rot;
    }
    if (w.moved_l[0]) {
        const Moved<R> m = moved_from<R>(r.pos, narrowq<R>(quat(r.rot)), r.start_pos, r.start_rot);
        put_moved(w, 0, i, m);
        if (inv_mass == R(0)) put_moved(w, 1, i, m);
    }
}

template <class P, class R>
__global__ void __launch_bounds__(256) k_init(DevWorld<P, R> w, uint32_t lo, uint32_t hi, SolveParams<R> o) {
    pdl_enter();
    for (uint32_t i = lo + blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += gridDim.x * blockDim.x)
        init_body(w, i, o);
}

// Where the primal and the dual find poses.  pos: a position; rot: a body's
// own rotation; rot_r: a rotation rounded to R; moved: what rows take; store:
// a body's new pose; careful, be_careful: solve6's hint.
// PoseFetch: pose buffer rd in global memory, displacements formed here.
template <class P, class R>
struct PoseFetch {
    const DevWorld<P, R>& w;
    int rd;
    __device__ __forceinline__ A4<P> pos(uint32_t j) const { return w.pos[rd][j]; }
    __device__ __forceinline__ A4<P> rot(uint32_t j) const { return w.rot[rd][j]; }
    __device__ __forceinline__ Q4<R> rot_r(uint32_t j) const { return narrowq<R>(quat(w.rot[rd][j])); }
    __device__ __forceinline__ A4<P> ipos(uint32_t j) const { return w.init_pos[j]; }
    __device__ __forceinline__ A4<P> irot(uint32_t j) const { return w.init_rot[j]; }
    __device__ __forceinline__ Moved<R> moved(uint32_t j) const {
        return moved_from<R>(w.pos[rd][j], rot_r(j), w.init_pos[j], w.init_rot[j]);
    }
};
// GlobalFetch: buffer rd read and wr written (the same buffer: in place, the
// coloured sweeps), displacements kept with the poses.
template <class P, class R>
struct GlobalFetch {
    const DevWorld<P, R>& w;
    int rd, wr;
    // warps that held a failing system this step, once they are an eighth of all
    __device__ __forceinline__ bool careful() const { return w.ctr->failed_solves > w.n_dyn / 256u; }
    __device__ __forceinline__ void be_careful() const {
        if ((threadIdx.x & 31u) == (uint32_t)__ffs(__activemask()) - 1u) atomicAdd(&w.ctr->failed_solves, 1u);
    }
    __device__ __forceinline__ A4<P> pos(uint32_t j) const { return w.pos[rd][j]; }
    __device__ __forceinline__ A4<P> rot(uint32_t j) const { return w.rot[rd][j]; }
    __device__ __forceinline__ Q4<R> rot_r(uint32_t j) const { return quat(w.rot_r[rd][j]); }
    __device__ __forceinline__ Moved<R> moved(uint32_t j) const {
        return moved_of(w.rot_r[rd][j], w.moved_l[rd][j], w.moved_a[rd][j]);
    }
    __device__ __forceinline__ void store(uint32_t i, A4<P> p, A4<P> q) const {
        const Moved<R> m = moved_from<R>(p, narrowq<R>(quat(q)), w.init_pos[i], w.init_rot[i]);
        w.pos[wr][i] = p;
        w.rot[wr][i] = q;
        put_moved(w, wr, i, m);
    }
};
// TileFetch: a shared-memory tile of consecutive bodies' poses, the others
// from global memory.
template <class P, class R, int T>
struct TileFetch {
    GlobalFetch<P, R> g;
    uint32_t lo;
    const A4<P>* sp;
    const A4<P>* sq;
    const A4<P>* si;
    const A4<P>* sr;
    __device__ __forceinline__ bool careful() const { return g.careful(); }
    __device__ __forceinline__ void be_careful() const { g.be_careful(); }
    __device__ __forceinline__ bool in(uint32_t j) const { return j - lo < (uint32_t)T; }
    __device__ __forceinline__ A4<P> pos(uint32_t j) const { return in(j) ? sp[j - lo] : g.pos(j); }
    __device__ __forceinline__ A4<P> rot(uint32_t j) const { return in(j) ? sq[j - lo] : g.rot(j); }
    __device__ __forceinline__ Q4<R> rot_r(uint32_t j) const {
        return in(j) ? narrowq<R>(quat(sq[j - lo])) : g.rot_r(j);
    }
    __device__ __forceinline__ Moved<R> moved(uint32_t j) const {
        return in(j) ? moved_from<R>(sp[j - lo], rot_r(j), si[j - lo], sr[j - lo]) : g.moved(j);
    }
    __device__ __forceinline__ void store(uint32_t i, A4<P> p, A4<P> q) const { g.store(i, p, q); }
};

// Clamped row forces shared by avbd_primal and avbd_dual (avbd/src/lib.rs:
// 380-406, 606-631): normal f0 <= 0, friction (f1, f2) scaled back onto the
// cone |f_t| <= mu |f0|; `tm` (unclamped friction magnitude) and `bounds`
// feed the dual's penalty rule.
template <class P>
__device__ __forceinline__ void row_forces(const RowDual<P, P>& du, P mu, P c0, P c1, P c2, P& f0, P& f1, P& f2,
                                           P& tm, P& bounds) {
    f0 = fmin_(du.penalty.x * c0 + du.lambda.x, P(0));
    const P f1r = du.penalty.y * c1 + du.lambda.y;
    const P f2r = du.penalty.z * c2 + du.lambda.z;
    bounds = dabs(f0) * mu;
    f1 = f1r;
    f2 = f2r;
    tm = dsqrt(f1r * f1r + f2r * f2r);
    if (tm > bounds && tm > P(0)) {
        const P s = bounds / tm;
        f1 = f1r * s;
        f2 = f2r * s;
    }
}

// The same in the split mode (FP64 forces, FP32 elsewhere): the cone
// magnitude tm and its scale factor in FP32, applied to the FP64 forces
// (lambda accumulates in FP64).  f0_neg: f0 < 0; inside: tm <= mu |f0|.
// FP64 instructions are few: the sign of f0 and the cone test are decided on
// bits and in FP32 (the rounded bound is within 2^-22 of the FP64 one)
// unless they are too close, tiny, or not finite.
__device__ __forceinline__ void row_forces_split(const RowDual<double, float>& du, float mu, float c0, float c1,
                                                 float c2, double& f0, double& f1, double& f2, bool& f0_neg,
                                                 bool& inside) {
    const double g0 = widen(du.penalty.x * c0) + du.lambda.x;
    const uint32_t hi = (uint32_t)__double2hiint(g0), lo = (uint32_t)__double2loint(g0), m = hi & 0x7FFFFFFFu;
    if (m >= 0x7FF00000u || (m | lo) == 0u) {  // infinite, NaN or zero
        f0 = fmin(g0, 0.0);
        f0_neg = f0 < 0.0;
    } else {
        f0_neg = hi >> 31;
        f0 = f0_neg ? g0 : 0.0;
    }
    const double f1r = widen(du.penalty.y * c1) + du.lambda.y;
    const double f2r = widen(du.penalty.z * c2) + du.lambda.z;
    f1 = f1r;
    f2 = f2r;
    const float f1q = to_float(f1r), f2q = to_float(f2r);
    const float tm = dsqrt(f1q * f1q + f2q * f2q);
    const float f0q = to_float(f0);
    const float bound = fabsf(f0q) * mu;
    bool outside;
    if (!f0_neg && f0q == 0.f && isfinite(mu) && !isnan(tm)) {  // f0 is a zero: so is the bound
        outside = tm > 0.f;
        inside = !outside;
    } else if (bound >= 1e-30f && bound <= 1e30f && tm >= bound * 1.000001f) {
        outside = true;
        inside = false;
    } else if (bound >= 1e-30f && bound <= 1e30f && tm <= bound * 0.999999f) {
        outside = false;
        inside = true;
    } else {
        const double b = fabs(f0) * (double)mu, t = (double)tm;
        outside = t > b && t > 0.0;
        inside = t <= b;
    }
    if (outside) {
        const float s = to_float(fabs(f0) * widen(mu)) / tm;
        f1 = f1r * widen(s);
        f2 = f2r * widen(s);
    }
}

// One contact row seen from body i (avbd/src/lib.rs:321-418): its three
// stamps (normal, tangent 1, tangent 2) as Jacobian rows (jl, ja), stiffness
// k and force f.
template <class R, class F>
__device__ __forceinline__ void primal_row_terms(const RowStatic<R>& rs, const RowDual<R, R>& du, uint32_t oth,
                                                 const F& fetch, Q4<R> sqr, V3<R> dqsl, V3<R> dqsa, R k_alpha,
                                                 V3<R> jl[3], V3<R> ja[3], R k[3], R f[3]) {
    const bool container = oth == kContainer;
    const bool is_a = container || !(oth & kIsB);
    const uint32_t other = oth & ~kIsB;
    V3<R> n = xyz(rs.n), t1 = xyz(rs.t1), t2 = xyz(rs.t2);
    V3<R> r0 = is_a ? n : neg(n);
    V3<R> r1 = is_a ? t1 : neg(t1);
    V3<R> r2 = is_a ? t2 : neg(t2);
    V3<R> rw = rotate(sqr, is_a ? xyz(rs.ra) : xyz(rs.rb));
    V3<R> dol{R(0), R(0), R(0)}, doa{R(0), R(0), R(0)}, rot_other{R(0), R(0), R(0)};
    if (!container) {
        const Moved<R> m = fetch.moved(other);
        dol = m.dl;
        doa = m.da;
        rot_other = rotate(m.q, is_a ? xyz(rs.rb) : xyz(rs.ra));
    }
    V3<R> j0 = cross(rw, r0), j1 = cross(rw, r1), j2 = cross(rw, r2);
    R c0 = rs.ra.w * k_alpha, c1 = rs.rb.w * k_alpha, c2 = rs.t1.w * k_alpha;
    c0 = c0 + (dot(r0, dqsl) + dot(j0, dqsa) - dot(r0, dol) - dot(cross(rot_other, r0), doa));
    c1 = c1 + (dot(r1, dqsl) + dot(j1, dqsa) - dot(r1, dol) - dot(cross(rot_other, r1), doa));
    c2 = c2 + (dot(r2, dqsl) + dot(j2, dqsa) - dot(r2, dol) - dot(cross(rot_other, r2), doa));
    // the forces only feed the R Hessian: in the split mode they are formed
    // in R from the rounded lambda (the dual accumulates lambda in P)
    R tm, bounds;
    row_forces(du, rs.n.w, c0, c1, c2, f[0], f[1], f[2], tm, bounds);
    jl[0] = r0;
    jl[1] = r1;
    jl[2] = r2;
    ja[0] = j0;
    ja[1] = j1;
    ja[2] = j2;
    k[0] = du.penalty.x;
    k[1] = du.penalty.y;
    k[2] = du.penalty.z;
}
template <class P, class R, class F>
__device__ __forceinline__ void primal_row_f(const DevWorld<P, R>& w, uint32_t r, uint32_t oth, const F& fetch,
                                             Q4<R> sqr, V3<R> dqsl, V3<R> dqsa, R k_alpha, Block6<R>& B) {
    V3<R> jl[3], ja[3];
    R k[3], f[3];
    primal_row_terms<R>(w.rs[r], w.rd.rounded(r), oth, fetch, sqr, dqsl, dqsa, k_alpha, jl, ja, k, f);
#pragma unroll
    for (int s = 0; s < 3; ++s) stamp(B, jl[s], ja[s], k[s], f[s]);
}

// One joint seen from body i (avbd/src/lib.rs:425-537).
template <class P, class R>
__device__ __forceinline__ void primal_joint(const DevWorld<P, R>& w, const DioConstraint& jt, uint32_t i, int rd,
                                             V3<P> sp, Q4<P> sq, Q4<R> sqr, Block6<R>& B) {
    const bool is_a = jt.a == i;
    V3<R> anc_a{R(jt.anchor_a[0]), R(jt.anchor_a[1]), R(jt.anchor_a[2])};
    V3<R> anc_b{R(jt.anchor_b[0]), R(jt.anchor_b[1]), R(jt.anchor_b[2])};
    V3<P> pa = is_a ? sp : xyz(w.pos[rd][jt.a]);
    V3<P> pb = !is_a ? sp : xyz(w.pos[rd][jt.b]);
    Q4<P> qa = is_a ? sq : quat(w.rot[rd][jt.a]);
    Q4<P> qb = !is_a ? sq : quat(w.rot[rd][jt.b]);
    V3<P> wpa = add(pa, rotate(qa, cast3<P>(anc_a)));
    V3<P> wpb = add(pb, rotate(qb, cast3<P>(anc_b)));
    V3<R> self_anchor = is_a ? anc_a : anc_b;
    R sign = is_a ? R(1) : R(-1);
    V3<R> delta = cast3<R>(sub(wpa, wpb));
    V3<R> r_self = rotate(sqr, self_anchor);
    R stiff = R(jt.anchor_b[3]);
    if (jt.kind == DIO_CONSTRAINT_BALL_SOCKET) {
        V3<R> jx = scale(V3<R>{R(1), R(0), R(0)}, sign);
        V3<R> jy = scale(V3<R>{R(0), R(1), R(0)}, sign);
        V3<R> jz = scale(V3<R>{R(0), R(0), R(1)}, sign);
        stamp(B, jx, cross(r_self, jx), stiff, delta.x * stiff);
        stamp(B, jy, cross(r_self, jy), stiff, delta.y * stiff);
        stamp(B, jz, cross(r_self, jz), stiff, delta.z * stiff);
    } else {
        R len = length(delta);
        R target = R(jt.anchor_a[3]);
        bool active = len > R(1.0e-6) && (jt.kind != DIO_CONSTRAINT_ROPE || len > target);
        if (active) {
            R dn[3] = {delta.x, delta.y, delta.z};
            divide_all(Pivot<R>(len), dn);  // the IEEE quotients (div_rn.cuh)
            const V3<R> nn{dn[0], dn[1], dn[2]};
            V3<R> jl = scale(nn, sign);
            V3<R> ja = cross(r_self, jl);
            stamp(B, jl, ja, stiff, stiff * (len - target));
        }
    }
}

// The same joint row from a JView: p_a - p_b is formed exactly as the
// reference forms it (joint a's anchor point minus joint b's).  `op4`/`oq`
// are the other body's snapshot pose, loaded by the caller.
template <class P, class R>
__device__ __forceinline__ void primal_jview_p(const JView& jv, A4<P> op4, Q4<R> oq, V3<P> sp, Q4<R> sqr,
                                               Block6<R>& B) {
    const bool is_a = !(jv.kind & kIsB);
    const uint32_t kind = jv.kind & ~kIsB;
    const V3<R> anc_s{R(jv.self_anchor.x), R(jv.self_anchor.y), R(jv.self_anchor.z)};
    const V3<R> anc_o{R(jv.other_anchor.x), R(jv.other_anchor.y), R(jv.other_anchor.z)};
    const V3<R> r_self = rotate(sqr, anc_s);
    V3<R> delta;  // joint a's anchor point minus joint b's
    if constexpr (std::is_same<P, R>::value) {
        const V3<P> p_self = add(sp, r_self);
        const V3<P> p_other = add(xyz(op4), rotate(oq, anc_o));
        delta = is_a ? sub(p_self, p_other) : sub(p_other, p_self);
    } else {
        // split mode: the position difference in P, the anchor offsets (small
        // body-frame vectors) rotated and differenced in R
        const V3<R> r_other = rotate(oq, anc_o);
        delta = is_a ? add(narrow3<R>(sub(sp, xyz(op4))), sub(r_self, r_other))
                     : add(narrow3<R>(sub(xyz(op4), sp)), sub(r_other, r_self));
    }
    const R sign = is_a ? R(1) : R(-1);
    const R stiff = R(jv.other_anchor.w);
    if (kind == DIO_CONSTRAINT_BALL_SOCKET) {
        V3<R> jx = scale(V3<R>{R(1), R(0), R(0)}, sign);
        V3<R> jy = scale(V3<R>{R(0), R(1), R(0)}, sign);
        V3<R> jz = scale(V3<R>{R(0), R(0), R(1)}, sign);
        if (finite_(stiff * (dabs(r_self.x) + dabs(r_self.y) + dabs(r_self.z)))) {
            stamp_masked<kMaskAxisX>(B, jx, cross(r_self, jx), stiff, delta.x * stiff);
            stamp_masked<kMaskAxisY>(B, jy, cross(r_self, jy), stiff, delta.y * stiff);
            stamp_masked<kMaskAxisZ>(B, jz, cross(r_self, jz), stiff, delta.z * stiff);
        } else {
            stamp(B, jx, cross(r_self, jx), stiff, delta.x * stiff);
            stamp(B, jy, cross(r_self, jy), stiff, delta.y * stiff);
            stamp(B, jz, cross(r_self, jz), stiff, delta.z * stiff);
        }
    } else {
        R len = length(delta);
        R target = R(jv.self_anchor.w);
        bool active = len > R(1.0e-6) && (kind != DIO_CONSTRAINT_ROPE || len > target);
        if (active) {
            R dn[3] = {delta.x, delta.y, delta.z};
            divide_all(Pivot<R>(len), dn);  // the IEEE quotients (div_rn.cuh)
            const V3<R> nn{dn[0], dn[1], dn[2]};
            V3<R> jl = scale(nn, sign);
            V3<R> ja = cross(r_self, jl);
            stamp(B, jl, ja, stiff, stiff * (len - target));
        }
    }
}

template <class P, class R, class F>
__device__ __forceinline__ void primal_jview_f(const JView& jv, const F& fetch, V3<P> sp, Q4<R> sqr, Block6<R>& B) {
    primal_jview_p<P, R>(jv, fetch.pos(jv.other), fetch.rot_r(jv.other), sp, sqr, B);
}

// What the primal of one body starts from besides its pose: its row list
// [j0, j0 + n), the diagonal m / dt^2, I / dt^2 and the inertial target.
template <class P, class R>
struct BodyTask {
    uint32_t i, j0, n;
    A4<R> mdt2;
    A4<P> ipos;
    A4<R> irot;
};

// The inertial start of a body's 6x6 system: diagonal M/dt^2, I/dt^2 and the
// gradient toward the inertial pose.
template <class P, class R>
__device__ __forceinline__ void primal_inertia(const BodyTask<P, R>& b, V3<P> sp, Q4<R> sqr, Block6<R>& B) {
    const R mdt2 = b.mdt2.x;
    const V3<R> idt2{b.mdt2.y, b.mdt2.z, b.mdt2.w};
#pragma unroll
    for (int k = 0; k < 21; ++k) B.h[k] = R(0);
    B.h[tri(0, 0)] = mdt2;
    B.h[tri(1, 1)] = mdt2;
    B.h[tri(2, 2)] = mdt2;
    B.h[tri(3, 3)] = idt2.x;
    B.h[tri(4, 4)] = idt2.y;
    B.h[tri(5, 5)] = idt2.z;
    const V3<R> rl = mulv(V3<R>{mdt2, mdt2, mdt2}, narrow3<R>(sub(sp, xyz(b.ipos))));
    const V3<R> ra = mulv(idt2, ang_diff(sqr, quat(b.irot)));
    B.g[0] = rl.x;
    B.g[1] = rl.y;
    B.g[2] = rl.z;
    B.g[3] = ra.x;
    B.g[4] = ra.y;
    B.g[5] = ra.z;
}

// Where the primal finds its bodies' constants and joints.  WorldBodies: by
// body, through the row and joint CSRs.
template <class P, class R>
struct WorldBodies {
    static constexpr bool kAhead = false;
    const DevWorld<P, R>& w;
    const uint32_t* list;
    __device__ __forceinline__ BodyTask<P, R> load(uint32_t t) const {
        BodyTask<P, R> b;
        b.i = list[t];
        b.j0 = w.row_off[b.i];
        // a caller's offsets may step back: such a body has no rows
        const uint32_t j1 = w.row_off[b.i + 1];
        b.n = j1 > b.j0 ? j1 - b.j0 : 0u;
        b.mdt2 = w.mdt2[b.i];
        b.ipos = w.inert_pos[b.i];
        b.irot = w.inert_rot[b.i];
        return b;
    }
    __device__ __forceinline__ uint32_t joints(uint32_t, uint32_t i) const {
        return w.n_joints ? w.joint_off[i + 1] - w.joint_off[i] : 0u;
    }
    __device__ __forceinline__ JView joint(uint32_t, uint32_t i, uint32_t q) const {
        return w.jview[w.joint_off[i] + q];
    }
};
// ListBodies: by position in the dynamic-body list, where the scene-chunk
// solve keeps them (SolveList): a warp's bodies are consecutive positions, so
// all of a body's constants and its first two joints are coalesced loads
// that depend on nothing but the position.
template <class P, class R>
struct ListBodies {
    static constexpr bool kAhead = sizeof(P) == 4;
    const DevWorld<P, R>& w;
    __device__ __forceinline__ BodyTask<P, R> load(uint32_t t) const {
        BodyTask<P, R> b;
        b.i = w.dyn_list[t];
        const uint2 r = w.solve.rows[t];
        b.j0 = r.x;
        b.n = r.y;
        b.mdt2 = w.mdt2[t];
        b.ipos = w.inert_pos[t];
        b.irot = w.inert_rot[t];
        return b;
    }
    __device__ __forceinline__ uint32_t joints(uint32_t t, uint32_t) const {
        return w.n_joints ? w.solve.joints[t] : 0u;
    }
    __device__ __forceinline__ JView joint(uint32_t t, uint32_t i, uint32_t q) const {
        if (q >= kListJoints) return w.jview[w.joint_off[i] + q];
        JView v;
        const uint2 m = w.solve.joint_meta[q * w.solve.stride + t];
        v.self_anchor = w.solve.joint_self[q * w.solve.stride + t];
        v.other_anchor = w.solve.joint_other[q * w.solve.stride + t];
        v.other = m.x;
        v.kind = m.y;
        return v;
    }
};

// A body's joints: their number and, where S::kAhead, the first of them
// loaded ahead of the row terms (the scene-chunk solve: 1024 scenes 2610 ->
// 2553 us a pass; elsewhere, and for two joints, its registers cost more).
struct JointsAhead {
    uint32_t n = 0;
    JView first;
    template <class S>
    __device__ __forceinline__ void load(const S& bodies, uint32_t t, uint32_t i) {
        n = bodies.joints(t, i);
        if constexpr (S::kAhead)
            if (n) first = bodies.joint(t, i, 0);
    }
};

// Joint rows, the 6x6 solve and the pose update of body i (the tail of
// avbd_primal); t: its position for `bodies`
template <class P, class R, class F, class S>
__device__ __forceinline__ void primal_finish(const S& bodies, uint32_t t, uint32_t i, const F& fetch, V3<P> sp,
                                              Q4<P> sq, Q4<R> sqr, const JointsAhead& joints, Block6<R>& B) {
    for (uint32_t k = 0; k < joints.n; ++k) {
        const JView jv = S::kAhead && k == 0u ? joints.first : bodies.joint(t, i, k);
        primal_jview_f<P, R>(jv, fetch, sp, sqr, B);
    }
    R dx[6];
    solve6(B, dx, fetch);
    const A4<P> np = pack(add(sp, widen3<P>(V3<R>{dx[0], dx[1], dx[2]})));
    if constexpr (std::is_same<P, R>::value)
        fetch.store(i, np, packq(quat_step(sq, V3<P>{dx[3], dx[4], dx[5]})));
    else
        fetch.store(i, np, packq(quat_step_split<P, R>(sq, sqr, V3<R>{dx[3], dx[4], dx[5]})));
}

// a body's own rotation rounded to R
template <class R, class P, class F>
__device__ __forceinline__ Q4<R> own_rot_r(const F& fetch, uint32_t i, Q4<P> q) {
    if constexpr (std::is_same<P, R>::value)
        return q;
    else
        return fetch.rot_r(i);
}

// avbd_primal for one body: reads the snapshot through `fetch` and stores
// the new pose through it.
template <class P, class R, class F>
__device__ __forceinline__ void primal_body_f(const DevWorld<P, R>& w, uint32_t i, const SolveParams<R>& o,
                                              const F& fetch) {
    if (w.inv[i].w == R(0)) return;
    const WorldBodies<P, R> bodies{w, &i};
    const BodyTask<P, R> b = bodies.load(0);
    const V3<P> sp = xyz(fetch.pos(i));
    const Q4<P> sq = quat(fetch.rot(i));
    const Q4<R> sqr = own_rot_r<R>(fetch, i, sq);
    Block6<R> B;
    primal_inertia(b, sp, sqr, B);
    if (b.n) {
        // displacement since the step start: read only by contact rows
        const Moved<R> m = fetch.moved(i);
        const R k_alpha = R(1) - o.alpha;
        for (uint32_t j = b.j0; j < b.j0 + b.n; ++j)
            primal_row_f(w, w.row_idx[j], w.row_oth[j], fetch, sqr, m.dl, m.da, k_alpha, B);
    }
    JointsAhead joints;
    joints.load(bodies, 0u, i);
    primal_finish(bodies, 0u, i, fetch, sp, sq, sqr, joints, B);
}

template <class P, class R>
__device__ __forceinline__ void primal_body(const DevWorld<P, R>& w, uint32_t i, int rd, const SolveParams<R>& o) {
    primal_body_f(w, i, o, GlobalFetch<P, R>{w, rd, 1 - rd});
}

// Tile variant: the CTA's T consecutive bodies stage their snapshot and
// step-start poses in shared memory; neighbours inside the tile (chain links,
// nearby boxes) are read from there.  Jacobi only (buffer rd is read-only
// during the launch).
template <class P, class R, int T, int MINB>
__global__ void __launch_bounds__(T, MINB) k_primal_tile(DevWorld<P, R> w, int rd, int wr, SolveParams<R> o) {
    __shared__ A4<P> s_pos[T], s_rot[T], s_ipos[T], s_irot[T];
    pdl_enter();
    const uint32_t lo = blockIdx.x * T;
    const uint32_t i = lo + threadIdx.x;
    if (i < w.n) {
        s_pos[threadIdx.x] = w.pos[rd][i];
        s_rot[threadIdx.x] = w.rot[rd][i];
        s_ipos[threadIdx.x] = w.init_pos[i];
        s_irot[threadIdx.x] = w.init_rot[i];
    }
    __syncthreads();
    if (i < w.n) {
        primal_body_f(w, i, o, TileFetch<P, R, T>{{w, rd, wr}, lo, s_pos, s_rot, s_ipos, s_irot});
    }
}

// One thread per dynamic body (static bodies are never solved,
// avbd/src/lib.rs:280-282, so they are left out of the launch).
// BLOCK threads per CTA, at least MINB CTAs per SM (a register bound); the
// variants are chosen per world by the autotuner.
template <class P, class R, int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) k_primal(DevWorld<P, R> w, int rd, int wr, SolveParams<R> o) {
    pdl_enter();
    for (uint32_t t = blockIdx.x * BLOCK + threadIdx.x; t < w.n_dyn; t += gridDim.x * BLOCK)
        primal_body(w, w.dyn_list[t], rd, o);
}

// avbd_dual, avbd/src/lib.rs:565-663: the row's dual update from its bodies' new poses (a, and b unless the
// row is against a container) and step-start poses.
template <class P, class R>
__device__ __forceinline__ RowDual<P, R> dual_update(const RowStatic<R>& rs, RowDual<P, R> du, const Moved<R>& a,
                                                     bool has_b, const Moved<R>& b, const SolveParams<R>& o) {
    V3<R> dbl{R(0), R(0), R(0)}, dba{R(0), R(0), R(0)}, rbw{R(0), R(0), R(0)};
    if (has_b) {
        dbl = b.dl;
        dba = b.da;
        rbw = rotate(b.q, xyz(rs.rb));
    }
    V3<R> raw = rotate(a.q, xyz(rs.ra));
    V3<R> r0 = xyz(rs.n), r1 = xyz(rs.t1), r2 = xyz(rs.t2);
    const R k_alpha = R(1) - o.alpha;
    R c0 = rs.ra.w * k_alpha, c1 = rs.rb.w * k_alpha, c2 = rs.t1.w * k_alpha;
    c0 = c0 + (dot(r0, a.dl) + dot(cross(raw, r0), a.da) - dot(r0, dbl) - dot(cross(rbw, r0), dba));
    c1 = c1 + (dot(r1, a.dl) + dot(cross(raw, r1), a.da) - dot(r1, dbl) - dot(cross(rbw, r1), dba));
    c2 = c2 + (dot(r2, a.dl) + dot(cross(raw, r2), a.da) - dot(r2, dbl) - dot(cross(rbw, r2), dba));
    bool f0_neg, inside;
    if constexpr (std::is_same<P, R>::value) {
        P f0, f1, f2, tm, bounds;
        row_forces(du, rs.n.w, c0, c1, c2, f0, f1, f2, tm, bounds);
        du.lambda.x = f0;
        du.lambda.y = f1;
        du.lambda.z = f2;
        f0_neg = f0 < P(0);
        inside = tm <= bounds;
    } else {
        const RowDual<P, R> old = du;
        row_forces_split(old, rs.n.w, c0, c1, c2, du.lambda.x, du.lambda.y, du.lambda.z, f0_neg, inside);
    }
    if (f0_neg) du.penalty.x = fmin_(du.penalty.x + o.beta_lin * dabs(c0), o.penalty_max);
    if (inside) {
        du.penalty.y = fmin_(du.penalty.y + o.beta_lin * dabs(c1), o.penalty_max);
        du.penalty.z = fmin_(du.penalty.z + o.beta_lin * dabs(c2), o.penalty_max);
    }
    return du;
}
// A group of up to 32 bodies by one warp, for bodies with contact rows.  A
// thread per body walks its rows one dependent gather and one chain of sums
// after another (about 900 cycles a row), so the warp lasts as long as its
// body with the most rows, and a world of a few thousand bodies leaves most
// of the GPU idle.  Here lane b holds body b, and the group's incidences --
// the bodies' row lists one after another -- are taken 32 at a time, a lane
// each whatever its body: the lane forms the incidence's three stamps
// (Jacobian row, stiffness, force) and stages them in shared memory; then
// lane e < 27 adds entry e of each body's 6x6 system (21 Hessian terms, 6
// gradient terms, each product formed as stamp() forms it) over the body's
// incidences and stamps in the serial order.  The sums see the same terms in
// the same order as primal_body_f, so the bits are the same; joints, the
// 6x6 solve and the pose update follow with a lane per body again.
// The staged sums cost about three times the instructions of a row in a warp
// whose bodies have equally many rows, so they are taken when the longest
// list exceeds kGroupSerial times the rounds of 32 (else: a thread per body).
// Measured (us per primal launch, cold caches): 31.8 -> 15.1 on the
// 8,192-cube field (8 incidences a body, groups of 4), 22.8 -> 18.1 on the
// 50,000-body pile (under one incidence a body, clustered), 18.6 -> 15.3 on
// 715 stacks of 7 cubes.  Serial threshold 1, 2 or 3: equal within 1 %, but 1
// takes the split-precision brick wall (7 incidences a body, evenly spread)
// 3.90 -> 4.47 ms a step.  Four CTAs an SM (128 registers) against five (96,
// spills): the field's two steps 922 against 976 us, the pile's 1672 against
// 1657.  Half the bodies a warp (24 warps an SM): every case slower.
constexpr uint32_t kGroupSerial = 2;
constexpr int kGroupStage = 25;  // 3 stamps of (J[6], k, f) padded to an odd stride
constexpr int kGroupSums = 27;
template <class R>
__host__ __device__ constexpr size_t primal_group_words() {
    return (size_t)32 * (kGroupStage + kGroupSums);
}
constexpr int kPrimalGroupWarps = 4;
template <class R>
__host__ __device__ constexpr size_t primal_group_smem() {
    return (size_t)kPrimalGroupWarps * primal_group_words<R>() * sizeof(R);
}

// Bodies t0 .. t0 + nb of `bodies` (dynamic ones, nb <= 32), all lanes of the
// warp; stage: the warp's primal_group_words<R>() words of shared memory
// (kStaged false: none, rows always serial).
template <bool kStaged, class P, class R, class F, class S>
__device__ __forceinline__ void primal_group(const DevWorld<P, R>& w, const S& bodies, uint32_t t0, uint32_t nb,
                                             const SolveParams<R>& o, const F& fetch, R* stage, uint32_t lane) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    R* const sums = stage + 32 * kGroupStage;  // [body][27]
    const bool live = lane < nb;
    BodyTask<P, R> task;
    task.i = task.j0 = task.n = 0;
    V3<P> sp{P(0), P(0), P(0)};
    Q4<P> sq{P(0), P(0), P(0), P(1)};
    Block6<R> B;
    JointsAhead joints;
    if (live) {
        task = bodies.load(t0 + lane);
        joints.load(bodies, t0 + lane, task.i);
        sp = xyz(fetch.pos(task.i));
        sq = quat(fetch.rot(task.i));
    }
    const Q4<R> sqr = live ? own_rot_r<R>(fetch, task.i, sq) : Q4<R>{R(0), R(0), R(0), R(1)};
    if (live) primal_inertia(task, sp, sqr, B);
    const uint32_t i = task.i, j0 = task.j0, n = task.n;
    uint32_t incl = n;  // inclusive sums of the row counts
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t t = __shfl_up_sync(kAll, incl, off);
        if (lane >= (uint32_t)off) incl += t;
    }
    const uint32_t total = __shfl_sync(kAll, incl, 31);
    if (total) {
        const R k_alpha = R(1) - o.alpha;
        V3<R> dqsl{R(0), R(0), R(0)}, dqsa{R(0), R(0), R(0)};
        if (n) {
            const Moved<R> m = fetch.moved(i);
            dqsl = m.dl;
            dqsa = m.da;
        }
        if (!kStaged || __reduce_max_sync(kAll, n) <= kGroupSerial * ((total + 31u) / 32u)) {
            for (uint32_t j = j0; j < j0 + n; ++j)
                primal_row_f(w, w.row_idx[j], w.row_oth[j], fetch, sqr, dqsl, dqsa, k_alpha, B);
        } else {
            if (n) {
#pragma unroll
                for (int e = 0; e < 21; ++e) sums[lane * kGroupSums + e] = B.h[e];
#pragma unroll
                for (int e = 0; e < 6; ++e) sums[lane * kGroupSums + 21 + e] = B.g[e];
            }
            // lane e's entry: H[ra][rb] (product J[ra] J[rb] k) or g[ra]
            // (J[ra] f 1, the 1 at the stride's last word)
            const bool is_h = lane < 21u;
            uint32_t ra = 0, rb = 7;
            stage[lane * kGroupStage + 24] = R(1);
            if (is_h) {
                while ((ra + 1) * (ra + 2) / 2 <= lane) ++ra;
                rb = lane - ra * (ra + 1) / 2;
            } else if (lane < (uint32_t)kGroupSums) {
                ra = lane - 21u;
            }
            for (uint32_t base = 0; base < total; base += 32u) {
                const uint32_t cnt = min(32u, total - base), f = base + lane;
                uint32_t s = 0;  // the incidence's body: the first with incl > f
#pragma unroll
                for (uint32_t step = 16; step; step >>= 1)
                    if (__shfl_sync(kAll, incl, s + step - 1) <= f) s += step;
                const uint32_t j = __shfl_sync(kAll, j0, s) + f - __shfl_sync(kAll, incl - n, s);
                auto from = [&](R v) { return __shfl_sync(kAll, v, s); };
                const Q4<R> q{from(sqr.x), from(sqr.y), from(sqr.z), from(sqr.w)};
                const V3<R> dl{from(dqsl.x), from(dqsl.y), from(dqsl.z)};
                const V3<R> da{from(dqsa.x), from(dqsa.y), from(dqsa.z)};
                if (lane < cnt) {
                    const uint32_t r = w.row_idx[j];
                    V3<R> jl[3], ja[3];
                    R k[3], ff[3];
                    primal_row_terms<R>(w.rs[r], w.rd.rounded(r), w.row_oth[j], fetch, q, dl, da, k_alpha, jl, ja, k,
                                        ff);
                    R* mine = stage + lane * kGroupStage;
#pragma unroll
                    for (int t = 0; t < 3; ++t) {
                        mine[t * 8 + 0] = jl[t].x;
                        mine[t * 8 + 1] = jl[t].y;
                        mine[t * 8 + 2] = jl[t].z;
                        mine[t * 8 + 3] = ja[t].x;
                        mine[t * 8 + 4] = ja[t].y;
                        mine[t * 8 + 5] = ja[t].z;
                        mine[t * 8 + 6] = k[t];
                        mine[t * 8 + 7] = ff[t];
                    }
                }
                __syncwarp();
                const uint32_t b1 = __shfl_sync(kAll, s, cnt - 1u);
                for (uint32_t b = __shfl_sync(kAll, s, 0); b <= b1; ++b) {
                    const uint32_t end = __shfl_sync(kAll, incl, b), cb = __shfl_sync(kAll, n, b);
                    const uint32_t q0 = max(end - cb, base) - base, q1 = min(end - base, cnt);
                    if (cb && lane < (uint32_t)kGroupSums) {
                        R acc = sums[b * kGroupSums + lane];
#pragma unroll 4
                        for (uint32_t t = q0; t < q1; ++t) {
                            const R* p = stage + t * kGroupStage;
                            R v[3];
#pragma unroll
                            for (uint32_t u = 0; u < 3; ++u)
                                v[u] = p[u * 8 + ra] * p[u * 8 + rb] * p[is_h ? u * 8 + 6 : 24];
#pragma unroll
                            for (uint32_t u = 0; u < 3; ++u) acc = acc + v[u];
                        }
                        sums[b * kGroupSums + lane] = acc;
                    }
                }
                __syncwarp();
            }
            if (n) {
#pragma unroll
                for (int e = 0; e < 21; ++e) B.h[e] = sums[lane * kGroupSums + e];
#pragma unroll
                for (int e = 0; e < 6; ++e) B.g[e] = sums[lane * kGroupSums + 21 + e];
            }
            __syncwarp();  // the next group's sums
        }
    }
    if (live) {
        primal_finish(bodies, t0 + lane, i, fetch, sp, sq, sqr, joints, B);
    }
}

// Worlds of jointed bodies: they carry few rows, and their joints are spread
// evenly by the list's order, so a thread per body is the better shape (the
// 257-scene split batch: 2.21 ms a pass against 2.27 in groups).
template <class P, class R>
inline bool mostly_jointed(const DevWorld<P, R>& w) { return (uint64_t)w.n_joints * 2 > w.n_dyn; }

// Bodies per warp: all 32 lanes once that gives every SM 12 warps, fewer
// (down to one) in smaller worlds, which would leave SMs idle.
inline uint32_t primal_group_size(uint32_t n_dyn, int sms) {
    uint32_t g = 32;
    while (g > 1 && n_dyn / g < (uint32_t)sms * 12u) g /= 2;
    return g;
}

template <class P, class R, class F>
__device__ __forceinline__ void primal_groups(const DevWorld<P, R>& w, const uint32_t* list, uint32_t n, uint32_t g,
                                              const SolveParams<R>& o, const F& fetch) {
    extern __shared__ __align__(16) unsigned char primal_group_smem_raw[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    R* stage = reinterpret_cast<R*>(primal_group_smem_raw) + warp * primal_group_words<R>();
    for (uint32_t t = (blockIdx.x * kPrimalGroupWarps + warp) * g; t < n; t += gridDim.x * kPrimalGroupWarps * g)
        primal_group<true>(w, WorldBodies<P, R>{w, list}, t, min(g, n - t), o, fetch, stage, lane);
}
template <class P, class R>
__global__ void __launch_bounds__(kPrimalGroupWarps * 32, sizeof(R) == 4 ? 4 : 2)
    k_primal_group(DevWorld<P, R> w, int rd, uint32_t g, SolveParams<R> o) {
    pdl_enter();
    primal_groups(w, w.dyn_list, w.n_dyn, g, o, GlobalFetch<P, R>{w, rd, 1 - rd});
}

// variants: 0-4 k_primal over the dynamic-body list with {threads per CTA,
// min CTAs per SM}; 5 (the default) k_primal_group, or k_primal in worlds of
// jointed bodies; 6-9 k_primal_tile over body tiles; 10 k_primal_group with a
// warp per body
constexpr int kPrimalVariants = DIO_PRIMAL_VARIANTS;

template <class P, class R>
inline void launch_primal(int variant, bool pdl, const DevWorld<P, R>& w, int rd, int wr, const SolveParams<R>& o,
                          int sms, cudaStream_t s) {
    const uint32_t nd = w.n_dyn > 0 ? w.n_dyn : 1;
    auto grid = [&](int block) { return grid_for(nd, block); };
    auto group = [&](uint32_t g) {
        launch_k(pdl, k_primal_group<P, R>, grid_for(nd, kPrimalGroupWarps * (int)g), kPrimalGroupWarps * 32,
                 primal_group_smem<R>(), s, w, rd, g, o);
    };
    switch (variant) {
        case 0:
            launch_k(pdl, k_primal<P, R, 128, 4>, grid(128), 128, 0, s, w, rd, wr, o);
            break;
        case 2:
            launch_k(pdl, k_primal<P, R, 128, 6>, grid(128), 128, 0, s, w, rd, wr, o);
            break;
        case 3:
            launch_k(pdl, k_primal<P, R, 256, 2>, grid(256), 256, 0, s, w, rd, wr, o);
            break;
        case 4:
            launch_k(pdl, k_primal<P, R, 256, 3>, grid(256), 256, 0, s, w, rd, wr, o);
            break;
        case 5:
            if (mostly_jointed(w))
                launch_k(pdl, k_primal<P, R, 64, 10>, grid(64), 64, 0, s, w, rd, wr, o);
            else
                group(primal_group_size(nd, sms));
            break;
        case 6:
            launch_k(pdl, k_primal_tile<P, R, 128, 5>, grid_for(w.n, 128), 128, 0, s, w, rd, wr, o);
            break;
        case 7:
            launch_k(pdl, k_primal_tile<P, R, 128, 6>, grid_for(w.n, 128), 128, 0, s, w, rd, wr, o);
            break;
        case 8:
            launch_k(pdl, k_primal_tile<P, R, 256, 3>, grid_for(w.n, 256), 256, 0, s, w, rd, wr, o);
            break;
        case 9:
            launch_k(pdl, k_primal_tile<P, R, 64, 10>, grid_for(w.n, 64), 64, 0, s, w, rd, wr, o);
            break;
        case 10:
            group(1);
            break;
        default:
            launch_k(pdl, k_primal<P, R, 128, 5>, grid(128), 128, 0, s, w, rd, wr, o);
            break;
    }
}

// Coloured Gauss-Seidel sweep: bodies color_order[c0 .. c1) in place, grouped
// or (worlds of jointed bodies, as in launch_primal) a thread each.
template <class P, class R>
__global__ void __launch_bounds__(kPrimalGroupWarps * 32, sizeof(R) == 4 ? 4 : 2)
    k_primal_color(DevWorld<P, R> w, uint32_t c0, uint32_t c1, uint32_t g, SolveParams<R> o) {
    primal_groups(w, w.color_order + c0, c1 - c0, g, o, GlobalFetch<P, R>{w, 0, 0});
}
template <class P, class R>
__global__ void __launch_bounds__(128)
    k_primal_color_bodies(DevWorld<P, R> w, uint32_t c0, uint32_t c1, SolveParams<R> o) {
    for (uint32_t t = c0 + blockIdx.x * blockDim.x + threadIdx.x; t < c1; t += gridDim.x * blockDim.x)
        primal_body_f(w, w.color_order[t], o, GlobalFetch<P, R>{w, 0, 0});
}

// avbd_dual, avbd/src/lib.rs:565-663, for row c; `fetch` reads the new state.
template <class P, class R, class F>
__device__ __forceinline__ void dual_row_f(const DevWorld<P, R>& w, uint32_t c, const F& fetch,
                                           const SolveParams<R>& o) {
    const uint2 ab = w.ab[c];
    const bool has_b = ab.y != kContainer;
    Moved<R> b{};
    if (has_b) b = fetch.moved(ab.y);
    w.rd.put(c, dual_update<P, R>(w.rs[c], w.rd[c], fetch.moved(ab.x), has_b, b, o));
}
template <class P, class R>
__device__ __forceinline__ void dual_row(const DevWorld<P, R>& w, uint32_t c, int rd, const SolveParams<R>& o) {
    dual_row_f(w, c, GlobalFetch<P, R>{w, rd, rd}, o);
}

template <class P, class R>
__global__ void __launch_bounds__(256) k_dual(DevWorld<P, R> w, uint32_t lo, uint32_t hi, const uint32_t* dyn_hi,
                                              int rd, SolveParams<R> o) {
    pdl_enter();
    uint32_t end = dyn_hi ? *dyn_hi : hi;
    for (uint32_t c = lo + blockIdx.x * blockDim.x + threadIdx.x; c < end; c += gridDim.x * blockDim.x)
        dual_row(w, c, rd, o);
}

// avbd_recover, avbd/src/lib.rs:667-699; also leaves the final pose in
// buffer 0 when it lives in buffer 1.
template <class P, class R, class F>
__device__ __forceinline__ void recover_body_f(const DevWorld<P, R>& w, uint32_t i, const F& fetch,
                                               const SolveParams<R>& o) {
    if (w.inv[i].w == R(0)) return;
    A4<P> p4 = fetch.pos(i);
    A4<P> q4 = fetch.rot(i);
    P dt = P(o.dt);
    A4<P> v = w.vel[i];
    w.prev_vel[i] = v;
    const Q4<P> rel = qmul(quat(q4), conj(quat(fetch.irot(i))));
    V3<P> nv, na;
    if constexpr (std::is_same<P, R>::value) {
        nv = divs(sub(xyz(p4), xyz(fetch.ipos(i))), dt);
        na = divs(V3<P>{P(2) * rel.x, P(2) * rel.y, P(2) * rel.z}, dt);
    } else {  // split mode: one division, then products (within an ulp of P)
        const P inv_dt = P(1) / dt;
        nv = scale(sub(xyz(p4), xyz(fetch.ipos(i))), inv_dt);
        na = scale(V3<P>{P(2) * rel.x, P(2) * rel.y, P(2) * rel.z}, inv_dt);
    }
    w.vel[i] = pack(nv);
    w.ang[i] = pack(na);
    // a non-finite pose or velocity is reported (DIO_ERR_NONFINITE), as the
    // reference demos' constraint tracing reports it (demos/constraints/src/main.rs:24-60)
    if (w.ctr && !(finite_(nv.x) && finite_(nv.y) && finite_(nv.z) && finite_(na.x) && finite_(na.y) &&
                   finite_(na.z) && finite_(q4.w)))
        atomicOr(&w.ctr->error_flags, kErrNonFinite);
}
template <class P, class R>
__device__ __forceinline__ void recover_body(const DevWorld<P, R>& w, uint32_t i, int rb, const SolveParams<R>& o) {
    recover_body_f(w, i, PoseFetch<P, R>{w, rb}, o);
}

template <class P, class R>
__global__ void __launch_bounds__(256) k_recover(DevWorld<P, R> w, uint32_t lo, uint32_t hi, int rb, int final_buf,
                                                 SolveParams<R> o) {
    pdl_enter();
    for (uint32_t i = lo + blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += gridDim.x * blockDim.x) {
        recover_body(w, i, rb, o);
        if (final_buf != 0) {
            w.pos[0][i] = w.pos[final_buf][i];
            w.rot[0][i] = w.rot[final_buf][i];
        }
    }
}

}  // namespace dio
