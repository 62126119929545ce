/*
 * fdtd_adjoint.cu — gradient of a receiver-trace loss with respect to a
 * per-cell absorption field, by the discrete adjoint of the open-room step.
 *
 * Forward (the reference's update with its PML profile replaced by a per-cell
 * field a_c = alpha_c * dt, as csrc/kernels/acoustic_fdtd.cpp:64 and :387-389
 * store alpha per cell; damping as :469-476 and :536-561):
 *   p~^n       = p^n + s[n] e_src                                (source)
 *   v^{n+1/2}  = (v^{n-1/2} - vc G p~^n) (.) d,  d_f = 1 - (a_L + a_R)/2
 *   p^{n+1}    = (p~^n - bulk D v^{n+1/2}) (.) q,  q_c = 1 / (1 + a_c)
 *   y^n        = R p^{n+1}                                       (receivers)
 * with G the gradient (4th order on interior faces, 2nd order on the first
 * and last face, acoustic_fdtd.cpp:1099-1148) and D the divergence (4th order
 * with zero velocity outside the faces, :894-952).
 *
 * Reverse step n, given Lp = dL/dp~^{n+1} and Lv = dL/dv^{n+1/2} (partial,
 * through step n+1's velocity update) and r^n = dL/dy^n:
 *   lam  = Lp + R^T r^n ;  U = lam (.) q ;
 *          g_c -= q_c^2 lam_c z_c, z = p~^n - bulk D v^{n+1/2}              (k_adj_cells, C1)
 *   mu   = Lv - bulk D^T U ;  W = mu (.) d ;  E_f = mu_f y_f,
 *          y = v^{n-1/2} - vc G p~^n ;  Lv <- W                            (k_adj_faces)
 *   Lp  <- U - vc G^T W ;  g_c -= 1/2 sum_{faces f of c} E_f               (k_adj_cells, C2)
 * Gradients accumulate in double.  The forward is recomputed segment by
 * segment from checkpoints (p~^n and v^{n-1/2} every K steps) into K+1
 * device slots, so the reverse sweep reads every state it needs from HBM.
 * Launches per step: forward and recompute 2 (velocity, which records the
 * receivers of the step before, and pressure, which adds the next step's source
 * sample), reverse 2 (faces; the cell updates that end a step and begin the one
 * before it).
 * Each sweep (forward, forward with checkpoints, backward) is captured once
 * as a CUDA graph and replayed while its length and buffers stay the same:
 * a gradient evaluation is then two graph launches.
 *
 * All kernels are templated on the working type R (float: the product path;
 * double: for finite-difference checks).  Every operation is separately
 * rounded (no contraction), so the float forward equals the reference's
 * arithmetic on the same absorption field bit for bit.
 */
#include "acoustic_fdtd_b200.h"
#include "fdtd_internal.h"
#include "launch.h"

#include <algorithm>
#include <climits>
#include <cstring>
#include <vector>

namespace fdtd {
namespace adj {

__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float rrcp(float a) { return __frcp_rn(a); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double rsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double rrcp(double a) { return __drcp_rn(a); }

template <class R>
struct ACoef {
    R vc, bulk, c1, c2;
};

template <class R>
__device__ __forceinline__ R face_d(R aL, R aR) { return rsub(R(1), rmul(R(0.5), radd(aL, aR))); }
template <class R>
__device__ __forceinline__ R cell_q(R a) { return rrcp(radd(R(1), a)); }

#define ADJ_INDEX                                                        \
    const int k = blockIdx.x * blockDim.x + threadIdx.x;                 \
    const int j = blockIdx.y * blockDim.y + threadIdx.y;                 \
    const int i = blockIdx.z;                                            \
    if (k >= g.nz || j >= g.ny) return;                                  \
    const long long id = ((long long)i * g.ny + j) * g.sz + k;

// Four consecutive values at an index that is a multiple of 4 (rows start on
// 8-element boundaries, so the access is aligned).
template <class R>
__device__ __forceinline__ void ld4r(const R* p, long long i, R (&v)[4])
{
    if constexpr (sizeof(R) == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p + i);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
        const double2 x = *reinterpret_cast<const double2*>(p + i);
        const double2 y = *reinterpret_cast<const double2*>(p + i + 2);
        v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
    }
}
template <class R>
__device__ __forceinline__ void st4r(R* p, long long i, const R (&v)[4])
{
    if constexpr (sizeof(R) == 4) {
        *reinterpret_cast<float4*>(p + i) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
        *reinterpret_cast<double2*>(p + i) = make_double2(v[0], v[1]);
        *reinterpret_cast<double2*>(p + i + 2) = make_double2(v[2], v[3]);
    }
}

template <class R>
__device__ __forceinline__ void ld2r(const R* p, long long i, R& a, R& b)
{
    if constexpr (sizeof(R) == 4) {
        const float2 x = *reinterpret_cast<const float2*>(p + i);
        a = x.x; b = x.y;
    } else {
        const double2 x = *reinterpret_cast<const double2*>(p + i);
        a = x.x; b = x.y;
    }
}
// the four values at i when they exist, else zero (i stays inside the field)
template <class R>
__device__ __forceinline__ void ld4z(const R* p, long long i, bool exists, R (&v)[4])
{
    ld4r(p, i, v);
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = exists ? v[q] : R(0);
}

// Threads own four consecutive cells k0 .. k0+3 of a row; the (row, group) pairs
// of a plane are numbered over 1-D blocks, so that no lane idles when Nz/4 is not
// a multiple of the warp.  The passes are bound by the latency of L2 and memory:
// what a thread reads is loaded at once from addresses kept inside the field,
// what does not exist is selected away afterwards, and each kernel starts while
// the one before it drains.
#define ADJ4_INDEX                                                       \
    const int nq_ = (g.nz + 3) >> 2;                                     \
    const int t_ = blockIdx.x * blockDim.x + threadIdx.x;                \
    if (t_ >= g.ny * nq_) return;                                        \
    const int j = t_ / nq_;                                              \
    const int k0 = 4 * (t_ - j * nq_);                                   \
    const int i = blockIdx.y;                                            \
    const long long id = ((long long)i * g.ny + j) * g.sz + k0;

// Blocks of 128 threads; the blocks an SM shall hold, given with each kernel, are
// those of the least time: more warps in flight are worth a few spilled registers
// (128^3, a reverse step with its recompute: 4 blocks of the cell updates and 5 of
// the faces 67.5 us, 5 and 7 61.8, 6 and 7 60.5, 7 and 8 60.7; a forward step
// with 6 and 6 blocks 15.7, 7 and 8 15.2).
constexpr int kAdjThreads = 128;

// Gradient on the x or y faces of four cells from the values around them: 4th
// order on interior faces, 2nd order on the first and last.
template <class R>
__device__ __forceinline__ R grad1(const ACoef<R>& cf, R pm, R pc, R pr, R p2, bool fourth)
{
    const R d = rsub(pr, pc), w = radd(rmul(cf.c1, d), rmul(cf.c2, rsub(p2, pm)));
    return fourth ? w : d;
}

// The values of a cell field a face update reads along x (or y): at f-1, f, f+1
// and f+2 for face f of an axis with n cells and stride st; c = those at f.
template <class R>
struct Line {
    R m[4], r[4], s[4];
    __device__ __forceinline__ Line(const R* p, long long id, long long st, int f, int n)
    {
        ld4r(p, f > 0 ? id - st : id, m);
        ld4r(p, f < n - 1 ? id + st : id, r);
        ld4r(p, f < n - 2 ? id + 2 * st : id, s);
    }
};

// A cell field at k0-1 .. k0+5, zero outside the row; c = its four own values.
template <class R>
__device__ __forceinline__ void zrow(const R* f, long long id, int k0, int nz, const R (&c)[4], R (&e)[7])
{
    e[0] = k0 > 0 ? f[id - 1] : R(0);
#pragma unroll
    for (int q = 0; q < 4; ++q) e[q + 1] = c[q];
    e[5] = e[6] = R(0);
    if (k0 + 4 < nz) ld2r(f, id + 4, e[5], e[6]);
    if (k0 + 5 >= nz) e[6] = R(0);
}
// A face field at k0-2 .. k0+4, zero outside the row; c = its four own values.
template <class R>
__device__ __forceinline__ void zfaces(const R* f, long long id, int k0, int nz, const R (&c)[4], R (&e)[7])
{
    e[0] = e[1] = R(0);
    if (k0 >= 2) ld2r(f, id - 2, e[0], e[1]);
#pragma unroll
    for (int q = 0; q < 4; ++q) e[q + 2] = c[q];
    e[6] = k0 + 4 < nz ? f[id + 4] : R(0);
}

// Divergence of the four cells, zero velocity outside the faces.
template <class R>
__device__ __forceinline__ void div4(const Grid& g, const R* vx, const R* vy, const R* vz, long long id, int i,
                                     int j, int k0, const ACoef<R>& cf, R (&dv)[4])
{
    const long long P = g.plane, S = g.sz;
    R xp[4], xm[4], xpp[4], xmm[4], yp[4], ym[4], ypp[4], ymm[4], zc[4], ez[7];
    ld4z(vx, id, i < g.nx - 1, xp);
    ld4z(vx, i > 0 ? id - P : id, i > 0, xm);
    ld4z(vx, i < g.nx - 2 ? id + P : id, i < g.nx - 2, xpp);
    ld4z(vx, i > 1 ? id - 2 * P : id, i > 1, xmm);
    ld4z(vy, id, j < g.ny - 1, yp);
    ld4z(vy, j > 0 ? id - S : id, j > 0, ym);
    ld4z(vy, j < g.ny - 2 ? id + S : id, j < g.ny - 2, ypp);
    ld4z(vy, j > 1 ? id - 2 * S : id, j > 1, ymm);
    ld4r(vz, id, zc);
    zfaces(vz, id, k0, g.nz, zc, ez);
    const R z0 = R(0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = k0 + q;
        const R zp = (k < g.nz - 1) ? ez[q + 2] : z0, zpp = (k < g.nz - 2) ? ez[q + 3] : z0;
        const R d1 = radd(radd(rsub(xp[q], xm[q]), rsub(yp[q], ym[q])), rsub(zp, ez[q + 1]));
        const R d2 = radd(radd(rsub(xpp[q], xmm[q]), rsub(ypp[q], ymm[q])), rsub(zpp, ez[q]));
        dv[q] = radd(rmul(cf.c1, d1), rmul(cf.c2, d2));
    }
}

// The receivers of one step: 8 taps summed w0*p0 + w1*p1 + ... as
// acoustic_fdtd.cpp:1663-1676, of the pressure before the source sample that the
// step after it adds to cell src (its value without the sample is *raw).
template <class R>
struct Record {
    int n = 0;
    const long long* idx = nullptr;
    const R* w = nullptr;
    R* row = nullptr;
    long long src = -1;
    const R* raw = nullptr;
};
template <class R>
__device__ __forceinline__ void record_receivers(const Record<R>& rec, const R* p, int first, int stride)
{
    for (int r = first; r < rec.n; r += stride) {
        R v[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const long long c = rec.idx[8 * r + t];
            v[t] = rmul(rec.w[8 * r + t], c == rec.src ? *rec.raw : p[c]);
        }
        R s = v[0];
#pragma unroll
        for (int t = 1; t < 8; ++t) s = radd(s, v[t]);
        rec.row[r] = s;
    }
}
template <class R>
__global__ void k_record(const R* p, Record<R> rec)
{
    record_receivers(rec, p, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// Velocity update.  It also records the receivers of the step before (the
// pressure it reads), which as a kernel of its own was 3.3 us of a 128^3 step
// (a step of the forward sweep: 18.5 us then, 15.2 now; the bytes its two passes
// move, 56 a cell, take 17.9 at the measured copy rate: the fields stay in L2).
template <class R>
__global__ void __launch_bounds__(kAdjThreads, sizeof(R) == 4 ? 7 : 3)
k_fwd_vel(Grid g, ACoef<R> cf, const R* __restrict__ a, const R* __restrict__ p, const R* vin0, const R* vin1,
          const R* vin2, R* vout0, R* vout1, R* vout2, Record<R> rec)
{
    wait_previous();
    release_next();
    if (rec.n > 0)
        record_receivers(rec, p, (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x,
                         gridDim.x * gridDim.y * blockDim.x);
    ADJ4_INDEX
    const long long P = g.plane, S = g.sz;
    R ac[4], ax[4], ay[4], pc[4], vx[4], vy[4], vz[4], e[7];
    ld4r(p, id, pc);
    const Line<R> lx(p, id, P, i, g.nx), ly(p, id, S, j, g.ny);
    zrow(p, id, k0, g.nz, pc, e);
    ld4r(vin0, id, vx);
    ld4r(vin1, id, vy);
    ld4r(vin2, id, vz);
    ld4r(a, id, ac);
    ld4r(a, i < g.nx - 1 ? id + P : id, ax);
    ld4r(a, j < g.ny - 1 ? id + S : id, ay);
    const R az = k0 + 4 < g.nz ? a[id + 4] : R(0);
    const bool fx = i > 0 && i < g.nx - 2, fy = j > 0 && j < g.ny - 2;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = k0 + q;
        const R x = rmul(rsub(vx[q], rmul(cf.vc, grad1(cf, lx.m[q], pc[q], lx.r[q], lx.s[q], fx))), face_d(ac[q], ax[q]));
        const R y = rmul(rsub(vy[q], rmul(cf.vc, grad1(cf, ly.m[q], pc[q], ly.r[q], ly.s[q], fy))), face_d(ac[q], ay[q]));
        const R z = rmul(rsub(vz[q], rmul(cf.vc, grad1(cf, e[q], e[q + 1], e[q + 2], e[q + 3], k > 0 && k < g.nz - 2))),
                         face_d(ac[q], q < 3 ? ac[q + 1] : az));
        if (k < g.nz) {
            vx[q] = x;
            vy[q] = y;
        }
        if (k < g.nz - 1) vz[q] = z;
    }
    if (i < g.nx - 1) st4r(vout0, id, vx);
    if (j < g.ny - 1) st4r(vout1, id, vy);
    st4r(vout2, id, vz);
}

// dep >= 0: the next step's source sample sig[dep_n] is added to the new
// pressure of cell dep, as k_deposit would before that step; raw (if given)
// keeps the pressure without it for the receivers.
template <class R>
__global__ void __launch_bounds__(kAdjThreads, sizeof(R) == 4 ? 8 : 3)
k_fwd_pres(Grid g, ACoef<R> cf, const R* __restrict__ a, const R* __restrict__ p, const R* __restrict__ vx,
           const R* __restrict__ vy, const R* __restrict__ vz, R* __restrict__ pn, long long dep,
           const R* __restrict__ sig, int dep_n, R* __restrict__ raw)
{
    wait_previous();
    release_next();
    ADJ4_INDEX
    R dv[4], pc[4], ac[4], out[4];
    ld4r(p, id, pc);
    ld4r(a, id, ac);
    div4(g, vx, vy, vz, id, i, j, k0, cf, dv);
#pragma unroll
    for (int q = 0; q < 4; ++q)
        out[q] = (k0 + q < g.nz) ? rmul(rsub(pc[q], rmul(cf.bulk, dv[q])), cell_q(ac[q])) : R(0);
    if (dep >= id && dep < id + 4) {
        const R sv = sig[dep_n];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (dep == id + q) {
                if (raw) *raw = out[q];
                if (sv != R(0)) out[q] = radd(out[q], sv);
            }
    }
    st4r(pn, id, out);
}

// Source deposit into the (open) source cell before step n.
template <class R>
__global__ void k_deposit(R* p, long long src, const R* sig, int n)
{
    const R s = sig[n];
    if (s != R(0)) p[src] = radd(p[src], s);
}

__device__ __forceinline__ void ld4d(const double* p, long long i, double (&v)[4]) { ld4r<double>(p, i, v); }
__device__ __forceinline__ void st4d(double* p, long long i, const double (&v)[4]) { st4r<double>(p, i, v); }

// The receivers' adjoint sources, by cell: the distinct tap cells in
// ascending order, and for each its taps (8 r + t) in the order R^T adds them.
template <class R>
struct TapSources {
    int n = 0;                       // distinct tap cells (0: none)
    const long long* cell = nullptr;
    const int* plane = nullptr;      // [nx + 1]: the tap cells of plane i are plane[i] .. plane[i+1]-1
    const int* start = nullptr;      // [n + 1]
    const int* tap = nullptr;        // 8 r + t, ascending within a cell
    const R* w = nullptr;            // tap weights [8 n_rec]
    const R* rrow = nullptr;         // this step's receiver residuals [n_rec]
};

// lam = Lp + R^T r^n on the tap cells among the four of group id in plane i
template <class R>
__device__ __forceinline__ void add_residuals(const TapSources<R>& ts, int i, long long id, R (&l)[4])
{
    const int end = ts.plane[i + 1];
    for (int c = ts.plane[i]; c < end; ++c) {   // no tap in most planes
        const long long d = ts.cell[c] - id;
        if (d < 0 || d > 3) continue;
        for (int e = ts.start[c]; e < ts.start[c + 1]; ++e) {
            const int tp = ts.tap[e];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (d == q) l[q] = radd(l[q], rmul(ts.w[tp], ts.rrow[tp >> 3]));
        }
    }
}

// Transposed gradient of the four cells along x or y: cell t of an axis with n
// cells (faces 0 .. n-2).  Terms in the order t-1, t, t-2, t+1.
template <class R>
__device__ __forceinline__ void gradT4(const R* w, long long id, long long s, int t, int n, const ACoef<R>& cf,
                                       R (&out)[4])
{
    auto inner = [&](int f) { return f > 0 && f < n - 2; };
    R m[4], c[4], mm[4], r[4];
    ld4z(w, t > 0 ? id - s : id, t > 0, m);
    ld4z(w, id, t < n - 1, c);
    ld4z(w, t > 1 ? id - 2 * s : id, inner(t - 2), mm);
    ld4z(w, t < n - 1 ? id + s : id, inner(t + 1), r);
    const R cm = inner(t - 1) ? cf.c1 : R(1), cc = inner(t) ? cf.c1 : R(1);
#pragma unroll
    for (int q = 0; q < 4; ++q)
        out[q] = rsub(radd(rsub(radd(R(0), rmul(cm, m[q])), rmul(cc, c[q])), rmul(cf.c2, mm[q])), rmul(cf.c2, r[q]));
}

// The cell updates of the reverse sweep.  C2: those that end step n (Lp from U, W
// and the faces' E); C1: those that begin the step before it (U from Lp, z from
// that step's states).  Both touch only a cell's own Lp, U and gradient, so
// between two steps of a segment one pass does both: Lp stays in registers and
// the gradient is read and written once, so that a step moves 128 bytes a cell
// (cells 68, faces 60) in place of 152 (128^3, a reverse step with its recompute:
// 73.6 us as three kernels, 60.5 now).
template <class R, bool C2, bool C1>
__global__ void __launch_bounds__(kAdjThreads, sizeof(R) == 4 ? (C1 && C2 ? 6 : 5) : 2)
k_adj_cells(Grid g, ACoef<R> cf, R* __restrict__ u, const R* __restrict__ w0, const R* __restrict__ w1,
            const R* __restrict__ w2, const R* __restrict__ e0, const R* __restrict__ e1, const R* __restrict__ e2,
            R* __restrict__ lp, double* __restrict__ grad, const R* __restrict__ a, const R* __restrict__ pt,
            const R* __restrict__ vx, const R* __restrict__ vy, const R* __restrict__ vz, TapSources<R> ts)
{
    wait_previous();
    release_next();
    ADJ4_INDEX
    const long long P = g.plane, S = g.sz;
    double gr[4];
    R l[4];
    ld4d(grad, id, gr);
    if constexpr (C2) {
        R gx[4], gy[4], uc[4], wc[4], ew[7], ex[4], exm[4], ey[4], eym[4], ez[4];
        ld4r(u, id, uc);
        ld4z(e0, id, i < g.nx - 1, ex);
        ld4z(e0, i > 0 ? id - P : id, i > 0, exm);
        ld4z(e1, id, j < g.ny - 1, ey);
        ld4z(e1, j > 0 ? id - S : id, j > 0, eym);
        ld4r(e2, id, ez);
        const R ezm = k0 >= 1 ? e2[id - 1] : R(0);
        ld4r(w2, id, wc);
        zfaces(w2, id, k0, g.nz, wc, ew);   // W_z at k0-2 .. k0+4
        gradT4(w0, id, P, i, g.nx, cf, gx);
        gradT4(w1, id, S, j, g.ny, cf, gy);
        auto innerz = [&](int f) { return f > 0 && f < g.nz - 2; };
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = k0 + q;
            const R tm = rmul(innerz(k - 1) ? cf.c1 : R(1), ew[q + 1]);
            const R tc = rmul(innerz(k) ? cf.c1 : R(1), k < g.nz - 1 ? ew[q + 2] : R(0));
            const R tmm = rmul(cf.c2, innerz(k - 2) ? ew[q] : R(0)), tr = rmul(cf.c2, innerz(k + 1) ? ew[q + 3] : R(0));
            const R gz = rsub(radd(rsub(radd(R(0), tm), tc), tmm), tr);
            l[q] = k < g.nz ? rsub(uc[q], rmul(cf.vc, radd(radd(gx[q], gy[q]), gz))) : R(0);
            const double e = (double)ex[q] + (double)exm[q] + (double)ey[q] + (double)eym[q] +
                             (k < g.nz - 1 ? (double)ez[q] : 0.0) + (double)(q ? ez[q - 1] : ezm);
            if (k < g.nz) gr[q] -= 0.5 * e;
        }
        if constexpr (!C1) st4r(lp, id, l);
    } else {
        ld4r(lp, id, l);
    }
    if constexpr (C1) {
        R ac[4], ptc[4], dv[4], uo[4];
        ld4r(a, id, ac);
        ld4r(pt, id, ptc);
        if (ts.n > 0) add_residuals(ts, i, id, l);
        div4(g, vx, vy, vz, id, i, j, k0, cf, dv);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const R qq = cell_q(ac[q]);
            const R z = rsub(ptc[q], rmul(cf.bulk, dv[q]));
            uo[q] = k0 + q < g.nz ? rmul(l[q], qq) : R(0);
            if (k0 + q < g.nz) gr[q] -= (double)qq * (double)qq * (double)l[q] * (double)z;
        }
        st4r(u, id, uo);
    }
    st4d(grad, id, gr);
}

// mu = Lv - bulk D^T U, W = mu (.) d and E = mu y on every face of the four cells.
template <class R>
__global__ void __launch_bounds__(kAdjThreads, sizeof(R) == 4 ? 7 : 2)
k_adj_faces(Grid g, ACoef<R> cf, const R* __restrict__ a, const R* __restrict__ u, const R* __restrict__ pt,
            const R* __restrict__ vo0, const R* __restrict__ vo1, const R* __restrict__ vo2, R* lv0, R* lv1, R* lv2,
            R* __restrict__ e0, R* __restrict__ e1, R* __restrict__ e2)
{
    wait_previous();
    release_next();
    ADJ4_INDEX
    R ac[4], ptc[4], uc[4];
    ld4r(a, id, ac);
    ld4r(pt, id, ptc);
    ld4r(u, id, uc);
    // x and y faces
    auto faces = [&](long long s, int f, int n, const R* vo, R* lv, R* ef) {
        R ar[4], l[4], v[4], eo[4];
        const Line<R> lu(u, id, s, f, n), lq(pt, id, s, f, n);
        ld4r(a, f < n - 1 ? id + s : id, ar);
        ld4r(lv, id, l);
        ld4r(vo, id, v);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const R um = f >= 1 ? lu.m[q] : R(0), us = f <= n - 3 ? lu.s[q] : R(0);
            const R dt = radd(rmul(cf.c1, rsub(uc[q], lu.r[q])), rmul(cf.c2, rsub(um, us)));
            const R mu = rsub(l[q], rmul(cf.bulk, dt));
            const R y = rsub(v[q], rmul(cf.vc, grad1(cf, lq.m[q], ptc[q], lq.r[q], lq.s[q], f > 0 && f < n - 2)));
            l[q] = k0 + q < g.nz ? rmul(mu, face_d(ac[q], ar[q])) : l[q];
            eo[q] = k0 + q < g.nz ? rmul(mu, y) : R(0);
        }
        if (f < n - 1) {
            st4r(lv, id, l);
            st4r(ef, id, eo);
        }
    };
    faces(g.plane, i, g.nx, vo0, lv0, e0);
    faces(g.sz, j, g.ny, vo1, lv1, e1);
    // z faces: U and P at k0-1 .. k0+5, a at k0 .. k0+4
    R eu[7], ep[7], l[4], v[4], eo[4];
    zrow(u, id, k0, g.nz, uc, eu);
    zrow(pt, id, k0, g.nz, ptc, ep);
    const R a4 = k0 + 4 < g.nz ? a[id + 4] : R(0);
    ld4r(lv2, id, l);
    ld4r(vo2, id, v);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = k0 + q;
        // c1 (u[k] - u[k+1]) + c2 (u[k-1] - u[k+2]), zero outside
        const R um = k >= 1 ? eu[q] : R(0), upp = k <= g.nz - 3 ? eu[q + 3] : R(0);
        const R dt = radd(rmul(cf.c1, rsub(eu[q + 1], eu[q + 2])), rmul(cf.c2, rsub(um, upp)));
        const R mu = rsub(l[q], rmul(cf.bulk, dt));
        const R y = rsub(v[q], rmul(cf.vc, grad1(cf, ep[q], ep[q + 1], ep[q + 2], ep[q + 3], k > 0 && k < g.nz - 2)));
        l[q] = k < g.nz - 1 ? rmul(mu, face_d(ac[q], q < 3 ? ac[q + 1] : a4)) : l[q];
        eo[q] = k < g.nz - 1 ? rmul(mu, y) : R(0);
    }
    st4r(lv2, id, l);
    st4r(e2, id, eo);
}

// a (reference order, float or double) -> padded R array
template <class R, class T>
__global__ void k_load_a(Grid g, const T* __restrict__ src, R* __restrict__ dst)
{
    ADJ_INDEX
    dst[id] = (R)src[((long long)i * g.ny + j) * g.nz + k];
}

// padded double grad -> reference order (double)
__global__ void k_store_grad(Grid g, const double* __restrict__ src, double* __restrict__ dst)
{
    ADJ_INDEX
    dst[((long long)i * g.ny + j) * g.nz + k] = src[id];
}

}  // namespace adj
}  // namespace fdtd

using namespace fdtd;
using namespace fdtd::adj;

struct FdtdB200Adj {
    int dbl = 0, device = 0, K = 200;
    cudaStream_t stream = nullptr;
    Grid g{};
    int N = 0;
    double dt = 0;
    ACoef<float> c32{};
    ACoef<double> c64{};
    size_t eb = 4;                 // bytes per value of R
    void* a = nullptr;             // padded R
    // loss-mode state and checkpoints
    void *P0 = nullptr, *P1 = nullptr, *V0[3] = {};
    std::vector<void*> ckP, ckV;   // ckV holds 3 per checkpoint
    // segment slots: K+1 P and K+1 x 3 V
    std::vector<void*> sP, sV;
    // adjoint state
    void *Lp = nullptr, *U = nullptr, *Lv[3] = {}, *E[3] = {};
    double* grad = nullptr;
    double* grad_ref = nullptr;    // reference-order staging
    // source/receivers
    long long src = -1;
    void* sig = nullptr;           // R[n_sig]
    void* raw = nullptr;           // R: the source cell's pressure without the next sample
    int n_sig = 0;
    int n_rec = 0;
    long long* ridx = nullptr;
    void* rw = nullptr;            // R[8 n_rec]
    void* traces = nullptr;        // R[n_steps x n_rec]
    void* resid = nullptr;         // R[n_steps x n_rec]
    int n_tap_cells = 0;           // distinct receiver tap cells, sorted (TapSources)
    long long* tap_cell = nullptr;
    int* tap_start = nullptr;
    int* tap_plane = nullptr;
    int* tap_ord = nullptr;
    int trace_cap = 0;
    int fwd_steps = -1;            // steps of the last checkpointed forward
    std::vector<void*> allocs;
    long long launches = 0;
    // CUDA graphs of whole sweeps, replayed while the buffers they name live:
    // forward without / with checkpoints (keyed by steps), backward (keyed by steps)
    struct Sweep {
        cudaGraphExec_t exec = nullptr;
        int steps = -1;
        long long launches = 0;
    } fwd[2], bwd;
};

namespace {

#define ACK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) { record_cuda_error(e_, #x); return FDTD_ERR_CUDA; } } while (0)

// Zeroed memory that the handle frees; *p stays null when there is none.
int dalloc(FdtdB200Adj* h, void** p, size_t bytes)
{
    const cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
        *p = nullptr;
        record_cuda_error(e, "device memory of an adjoint handle");
        cudaGetLastError();   // or the next launch would report it
        return FDTD_ERR_CUDA;
    }
    h->allocs.push_back(*p);
    ACK(cudaMemsetAsync(*p, 0, bytes, h->stream));
    return FDTD_OK;
}

void dfree(FdtdB200Adj* h, void*& p)
{
    if (!p) return;
    cudaFree(p);
    h->allocs.erase(std::remove(h->allocs.begin(), h->allocs.end(), p), h->allocs.end());
    p = nullptr;
}

size_t field_bytes(const FdtdB200Adj* h) { return (size_t)h->g.cells * h->eb; }

dim3 cell_grid(const Grid& g) { return dim3((g.nz + 31) / 32, (g.ny + 7) / 8, g.nx); }
const dim3 kBlock(32, 8, 1);
dim3 vec_grid(const Grid& g)   // four cells per thread (ADJ4_INDEX)
{
    return dim3((unsigned)(((long long)g.ny * ((g.nz + 3) / 4) + kAdjThreads - 1) / kAdjThreads), g.nx);
}

template <class R>
const ACoef<R>& coef(const FdtdB200Adj* h);
template <>
const ACoef<float>& coef<float>(const FdtdB200Adj* h) { return h->c32; }
template <>
const ACoef<double>& coef<double>(const FdtdB200Adj* h) { return h->c64; }

// One forward step from (p, vin) to (pn, vout); p already holds this step's
// source sample.  The pressure kernel adds the next step's sample to pn
// (next_deposit).  rec: the receivers of p, the step before's, to record.
template <class R>
int fwd_step(FdtdB200Adj* h, int n, void* p, void* const* vin, void* const* vout, void* pn, bool next_deposit,
             const Record<R>& rec)
{
    const Grid& g = h->g;
    const ACoef<R>& cf = coef<R>(h);
    const bool dep = next_deposit && h->src >= 0 && n + 1 < h->n_sig;
    ACK(launch_after(k_fwd_vel<R>, vec_grid(g), dim3(kAdjThreads), 0, h->stream, g, cf, (const R*)h->a, (const R*)p,
                     (const R*)vin[0], (const R*)vin[1], (const R*)vin[2], (R*)vout[0], (R*)vout[1], (R*)vout[2], rec));
    ACK(launch_after(k_fwd_pres<R>, vec_grid(g), dim3(kAdjThreads), 0, h->stream, g, cf, (const R*)h->a, (const R*)p,
                     (const R*)vout[0], (const R*)vout[1], (const R*)vout[2], (R*)pn, dep ? h->src : -1LL,
                     (const R*)h->sig, n + 1, (R*)h->raw));
    h->launches += 2;
    return FDTD_OK;
}

// Four fields in one allocation: P, then the three velocities.  All or, when
// memory runs out, none.
int alloc_state(FdtdB200Adj* h, int count, std::vector<void*>& P, std::vector<void*>& V)
{
    const size_t step = (field_bytes(h) + 255) & ~(size_t)255;
    void* slab = nullptr;
    if (int rc = dalloc(h, &slab, 4 * step * count)) return rc;
    for (char* at = (char*)slab; count > 0; --count, at += 4 * step) {
        P.push_back(at);
        for (int c = 1; c <= 3; ++c) V.push_back(at + c * step);
    }
    return FDTD_OK;
}

int ensure_checkpoints(FdtdB200Adj* h, int n_steps)
{
    const int n_ck = (n_steps + h->K - 1) / h->K;
    while ((int)h->ckP.size() < n_ck)
        if (int rc = alloc_state(h, 1, h->ckP, h->ckV)) return rc;
    return FDTD_OK;
}

// The forward sweep (enqueued only; checkpoints must already exist).
template <class R>
int forward_impl(FdtdB200Adj* h, int n_steps, int keep)
{
    const size_t fb = field_bytes(h);
    ACK(cudaMemsetAsync(h->P0, 0, fb, h->stream));
    for (int c = 0; c < 3; ++c) ACK(cudaMemsetAsync(h->V0[c], 0, fb, h->stream));
    void* P[2] = {h->P0, h->P1};
    int cur = 0;
    Record<R> rec;   // of the step before: recorded as its pressure is read
    if (h->src >= 0 && h->n_sig > 0) {   // step 0's source sample; later ones come with the step before
        k_deposit<R><<<1, 1, 0, h->stream>>>((R*)P[cur], h->src, (const R*)h->sig, 0);
        ++h->launches;
    }
    for (int n = 0; n < n_steps; ++n) {
        if (keep && n % h->K == 0) {   // p~^n: P^n with its source sample
            const int q = n / h->K;
            ACK(cudaMemcpyAsync(h->ckP[q], P[cur], fb, cudaMemcpyDeviceToDevice, h->stream));
            for (int c = 0; c < 3; ++c)
                ACK(cudaMemcpyAsync(h->ckV[3 * q + c], h->V0[c], fb, cudaMemcpyDeviceToDevice, h->stream));
        }
        if (int rc = fwd_step<R>(h, n, P[cur], h->V0, h->V0, P[cur ^ 1], n + 1 < n_steps, rec)) return rc;
        cur ^= 1;
        if (h->n_rec > 0 && n < h->trace_cap) {
            rec.n = h->n_rec;
            rec.idx = h->ridx;
            rec.w = (const R*)h->rw;
            rec.row = (R*)h->traces + (size_t)n * h->n_rec;
            rec.src = n + 1 < n_steps && n + 1 < h->n_sig ? h->src : -1;
            rec.raw = (const R*)h->raw;
        }
    }
    if (rec.n > 0) {
        k_record<R><<<(rec.n + 127) / 128, 128, 0, h->stream>>>((const R*)P[cur], rec);
        ++h->launches;
    }
    ACK(cudaGetLastError());
    return FDTD_OK;
}

void drop_sweep(FdtdB200Adj::Sweep& g)
{
    if (g.exec) cudaGraphExecDestroy(g.exec);
    g = FdtdB200Adj::Sweep();
}

void drop_sweeps(FdtdB200Adj* h)
{
    drop_sweep(h->fwd[0]);
    drop_sweep(h->fwd[1]);
    drop_sweep(h->bwd);
}

// Replays the cached graph of a sweep, capturing it first when it is missing
// or was made for another length.  enqueue(h) issues the sweep on h->stream.
template <class F>
int run_sweep(FdtdB200Adj* h, FdtdB200Adj::Sweep& g, int steps, F enqueue)
{
    if (!g.exec || g.steps != steps) {
        drop_sweep(g);
        const long long l0 = h->launches;
        ACK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
        const int rc = enqueue(h);
        cudaGraph_t graph = nullptr;
        const cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
        if (rc) {
            if (graph) cudaGraphDestroy(graph);
            return rc;
        }
        ACK(e);
        const cudaError_t ei = cudaGraphInstantiate(&g.exec, graph, 0);
        cudaGraphDestroy(graph);
        ACK(ei);
        g.steps = steps;
        g.launches = h->launches - l0;
        h->launches = l0;
    }
    ACK(cudaGraphLaunch(g.exec, h->stream));
    h->launches += g.launches;
    return FDTD_OK;
}

int ensure_slots(FdtdB200Adj* h)
{
    const size_t fb = field_bytes(h);
    // the states of a longest segment, in one allocation (128^3, 200 steps: the first
    // backward pass takes 25 ms, 300 to 380 with an allocation for each field)
    const int need = std::min(h->K, h->fwd_steps) + 1, have = (int)h->sP.size();
    if (have < need)
        if (int rc = alloc_state(h, need - have, h->sP, h->sV)) return rc;
    // each of the sweep's own fields that an earlier try found no memory for, too
    void** const field[] = {&h->Lp, &h->U, &h->Lv[0], &h->Lv[1], &h->Lv[2], &h->E[0], &h->E[1], &h->E[2]};
    for (void** p : field)
        if (!*p)
            if (int rc = dalloc(h, p, fb)) return rc;
    if (!h->grad)
        if (int rc = dalloc(h, (void**)&h->grad, (size_t)h->g.cells * sizeof(double))) return rc;
    if (!h->grad_ref)
        if (int rc = dalloc(h, (void**)&h->grad_ref, (size_t)h->N * sizeof(double))) return rc;
    return FDTD_OK;
}

template <class R>
int backward_impl(FdtdB200Adj* h)
{
    const Grid& g = h->g;
    const ACoef<R>& cf = coef<R>(h);
    const size_t fb = field_bytes(h);
    const int n_steps = h->fwd_steps;
    ACK(cudaMemsetAsync(h->Lp, 0, fb, h->stream));
    for (int c = 0; c < 3; ++c) {
        ACK(cudaMemsetAsync(h->Lv[c], 0, fb, h->stream));
        ACK(cudaMemsetAsync(h->E[c], 0, fb, h->stream));
    }
    ACK(cudaMemsetAsync(h->grad, 0, (size_t)g.cells * sizeof(double), h->stream));
    const int n_seg = (n_steps + h->K - 1) / h->K;
    for (int s = n_seg - 1; s >= 0; --s) {
        const int n0 = s * h->K, n1 = std::min(n0 + h->K, n_steps), len = n1 - n0;
        ACK(cudaMemcpyAsync(h->sP[0], h->ckP[s], fb, cudaMemcpyDeviceToDevice, h->stream));
        for (int c = 0; c < 3; ++c)
            ACK(cudaMemcpyAsync(h->sV[c], h->ckV[3 * s + c], fb, cudaMemcpyDeviceToDevice, h->stream));
        // recompute: slot t holds p~^{n0+t} (after its deposit; the checkpoint
        // already holds it) and v^{n0+t-1/2}; traces are already recorded
        for (int t = 0; t < len; ++t)
            if (int rc = fwd_step<R>(h, n0 + t, h->sP[t], &h->sV[3 * t], &h->sV[3 * (t + 1)], h->sP[t + 1],
                                     t + 1 < len, Record<R>()))
                return rc;
        // cell updates: c2 those that end step n0 + t + 1, c1 those that begin step n0 + t
        auto cells = [&](auto kernel, int t) -> int {
            TapSources<R> ts;   // R^T r^n, added to Lp
            if (h->n_rec > 0 && t >= 0) {
                ts.n = h->n_tap_cells;
                ts.cell = h->tap_cell;
                ts.plane = h->tap_plane;
                ts.start = h->tap_start;
                ts.tap = h->tap_ord;
                ts.w = (const R*)h->rw;
                ts.rrow = (const R*)h->resid + (size_t)(n0 + t) * h->n_rec;
            }
            void* const* vn = &h->sV[3 * (std::max(t, 0) + 1)];   // v^{n+1/2}
            ACK(launch_after(kernel, vec_grid(g), dim3(kAdjThreads), 0, h->stream, g, cf, (R*)h->U, (const R*)h->Lv[0],
                             (const R*)h->Lv[1], (const R*)h->Lv[2], (const R*)h->E[0], (const R*)h->E[1],
                             (const R*)h->E[2], (R*)h->Lp, h->grad, (const R*)h->a, (const R*)h->sP[std::max(t, 0)],
                             (const R*)vn[0], (const R*)vn[1], (const R*)vn[2], ts));
            ++h->launches;
            return FDTD_OK;
        };
        for (int t = len - 1; t >= 0; --t) {
            if (int rc = t == len - 1 ? cells(k_adj_cells<R, false, true>, t) : cells(k_adj_cells<R, true, true>, t)) return rc;
            void* const* vo = &h->sV[3 * t];       // v^{n-1/2}
            ACK(launch_after(k_adj_faces<R>, vec_grid(g), dim3(kAdjThreads), 0, h->stream, g, cf, (const R*)h->a,
                             (const R*)h->U, (const R*)h->sP[t], (const R*)vo[0], (const R*)vo[1], (const R*)vo[2],
                             (R*)h->Lv[0], (R*)h->Lv[1], (R*)h->Lv[2], (R*)h->E[0], (R*)h->E[1], (R*)h->E[2]));
            ++h->launches;
        }
        if (int rc = cells(k_adj_cells<R, true, false>, -1)) return rc;
        ACK(cudaGetLastError());
    }
    return FDTD_OK;
}

template <class R>
void set_coef(ACoef<R>& cf, R dx, R c, R rho, R dt)
{
    cf.vc = dt / (rho * dx);
    const R inv_dx = R(1) / dx;
    cf.bulk = rho * c * c * dt * inv_dx;
    cf.c1 = R(9) / R(8);
    cf.c2 = R(-1) / R(24);
}

long long pad_index(const Grid& g, int flat)
{
    const int k = flat % g.nz, t = flat / g.nz, j = t % g.ny, i = t / g.ny;
    return ((long long)i * g.ny + j) * g.sz + k;
}

}  // namespace

extern "C" {

FdtdB200Adj* fdtd_b200_adj_create(int Nx, int Ny, int Nz, double dx, double c, double rho_air,
                                  int use_double, int checkpoint_every, int device)
{
    if (Nx < 1 || Ny < 1 || Nz < 1 || dx <= 0 || c <= 0 || checkpoint_every < 1) return nullptr;
    if ((long long)Nx * Ny * Nz > INT_MAX) return nullptr;
    FdtdB200Adj* h = new FdtdB200Adj();
    h->dbl = use_double ? 1 : 0;
    h->eb = h->dbl ? 8 : 4;
    h->K = checkpoint_every;
    if (device < 0) cudaGetDevice(&device);
    h->device = device;
    if (cudaSetDevice(device) != cudaSuccess ||
        cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete h;
        return nullptr;
    }
    Grid& g = h->g;
    g.nx = Nx; g.ny = Ny; g.nz = Nz;
    g.sz = (Nz + kRowAlign - 1) / kRowAlign * kRowAlign;
    g.plane = (long long)Ny * g.sz;
    g.cells = (long long)Nx * g.plane;
    h->N = Nx * Ny * Nz;
    // the reference's time step (acoustic_fdtd.cpp:345-349) in each working type
    const float dt32 = 0.77f * (float)dx / ((float)c * 1.732050808f);
    const double dt64 = 0.77 * dx / (c * 1.732050808);
    set_coef<float>(h->c32, (float)dx, (float)c, (float)rho_air, dt32);
    set_coef<double>(h->c64, dx, c, rho_air, dt64);
    h->dt = h->dbl ? dt64 : (double)dt32;
    const size_t fb = field_bytes(h);
    int rc = dalloc(h, &h->a, fb);
    if (!rc) rc = dalloc(h, &h->raw, h->eb);
    if (!rc) rc = dalloc(h, &h->P0, fb);
    if (!rc) rc = dalloc(h, &h->P1, fb);
    for (int q = 0; q < 3 && !rc; ++q) rc = dalloc(h, &h->V0[q], fb);
    if (!rc && cudaStreamSynchronize(h->stream) != cudaSuccess) rc = FDTD_ERR_CUDA;
    if (rc) {
        fdtd_b200_adj_destroy(h);
        return nullptr;
    }
    return h;
}

void fdtd_b200_adj_destroy(FdtdB200Adj* h)
{
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    drop_sweeps(h);
    for (void* p : h->allocs) cudaFree(p);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

double fdtd_b200_adj_dt(const FdtdB200Adj* h) { return h ? h->dt : 0.0; }

long long fdtd_b200_adj_launch_count(const FdtdB200Adj* h) { return h ? h->launches : 0; }

int fdtd_b200_adj_set_absorption(FdtdB200Adj* h, const void* a_cell, int len, int value_bytes)
{
    if (!h || !a_cell) return FDTD_ERR_NULL;
    if (len != h->N) return FDTD_ERR_DIM;
    if (value_bytes != 4 && value_bytes != 8) return FDTD_ERR_ARG;
    ACK(cudaSetDevice(h->device));
    void* stage = nullptr;
    ACK(cudaMallocAsync(&stage, (size_t)len * value_bytes, h->stream));
    cudaError_t e = cudaMemcpyAsync(stage, a_cell, (size_t)len * value_bytes, cudaMemcpyDefault, h->stream);
    if (e == cudaSuccess) {
        const Grid& g = h->g;
        if (h->dbl && value_bytes == 8)
            k_load_a<double, double><<<cell_grid(g), kBlock, 0, h->stream>>>(g, (const double*)stage, (double*)h->a);
        else if (h->dbl)
            k_load_a<double, float><<<cell_grid(g), kBlock, 0, h->stream>>>(g, (const float*)stage, (double*)h->a);
        else if (value_bytes == 8)
            k_load_a<float, double><<<cell_grid(g), kBlock, 0, h->stream>>>(g, (const double*)stage, (float*)h->a);
        else
            k_load_a<float, float><<<cell_grid(g), kBlock, 0, h->stream>>>(g, (const float*)stage, (float*)h->a);
        e = cudaGetLastError();
    }
    cudaFreeAsync(stage, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) {
        record_cuda_error(e, "fdtd_b200_adj_set_absorption");
        return FDTD_ERR_CUDA;
    }
    h->fwd_steps = -1;
    return FDTD_OK;
}

int fdtd_b200_adj_set_source(FdtdB200Adj* h, int cell, const double* signal, int n)
{
    if (!h) return FDTD_ERR_NULL;
    if (cell < 0 || cell >= h->N || n < 0 || (n > 0 && !signal)) return FDTD_ERR_ARG;
    ACK(cudaSetDevice(h->device));
    ACK(cudaStreamSynchronize(h->stream));
    drop_sweeps(h);
    dfree(h, h->sig);
    h->src = pad_index(h->g, cell);
    h->n_sig = 0;
    h->fwd_steps = -1;
    if (n > 0) {
        int rc = dalloc(h, &h->sig, (size_t)n * h->eb);
        if (rc) return rc;
        std::vector<unsigned char> buf((size_t)n * h->eb);
        for (int q = 0; q < n; ++q) {
            if (h->dbl) memcpy(&buf[(size_t)q * 8], &signal[q], 8);
            else { const float f = (float)signal[q]; memcpy(&buf[(size_t)q * 4], &f, 4); }
        }
        ACK(cudaMemcpyAsync(h->sig, buf.data(), buf.size(), cudaMemcpyHostToDevice, h->stream));
        ACK(cudaStreamSynchronize(h->stream));
    }
    h->n_sig = n;
    return FDTD_OK;
}

int fdtd_b200_adj_set_receivers(FdtdB200Adj* h, int n_rec, const int* idx8, const double* wgt8, int max_steps)
{
    if (!h || (n_rec > 0 && (!idx8 || !wgt8))) return FDTD_ERR_NULL;
    if (n_rec < 0 || max_steps < 0) return FDTD_ERR_ARG;
    std::vector<long long> pi((size_t)n_rec * 8);
    for (size_t q = 0; q < pi.size(); ++q) {
        if (idx8[q] < 0 || idx8[q] >= h->N) return FDTD_ERR_ARG;
        pi[q] = pad_index(h->g, idx8[q]);
    }
    ACK(cudaSetDevice(h->device));
    ACK(cudaStreamSynchronize(h->stream));
    drop_sweeps(h);
    void* ri = h->ridx;
    dfree(h, ri);
    h->ridx = nullptr;
    dfree(h, h->rw);
    dfree(h, h->traces);
    dfree(h, h->resid);
    {
        void* t1 = h->tap_cell;
        void* t2 = h->tap_start;
        void* t3 = h->tap_ord;
        dfree(h, t1);
        dfree(h, t2);
        dfree(h, t3);
        void* t4 = h->tap_plane;
        dfree(h, t4);
    }
    h->tap_plane = nullptr;
    h->tap_cell = nullptr;
    h->tap_start = nullptr;
    h->tap_ord = nullptr;
    h->n_tap_cells = 0;
    h->n_rec = h->trace_cap = 0;   // no forward runs until the new ones are complete
    h->fwd_steps = -1;
    if (n_rec > 0) {
        void* p = nullptr;
        int rc = dalloc(h, &p, pi.size() * sizeof(long long));
        if (rc) return rc;
        h->ridx = (long long*)p;
        rc = dalloc(h, &h->rw, pi.size() * h->eb);
        if (!rc) rc = dalloc(h, &h->traces, (size_t)std::max(max_steps, 1) * n_rec * h->eb);
        if (!rc) rc = dalloc(h, &h->resid, (size_t)std::max(max_steps, 1) * n_rec * h->eb);
        if (rc) return rc;
        std::vector<unsigned char> wb(pi.size() * h->eb);
        for (size_t q = 0; q < pi.size(); ++q) {
            if (h->dbl) memcpy(&wb[q * 8], &wgt8[q], 8);
            else { const float f = (float)wgt8[q]; memcpy(&wb[q * 4], &f, 4); }
        }
        ACK(cudaMemcpyAsync(h->ridx, pi.data(), pi.size() * sizeof(long long), cudaMemcpyHostToDevice, h->stream));
        ACK(cudaMemcpyAsync(h->rw, wb.data(), wb.size(), cudaMemcpyHostToDevice, h->stream));
        // taps grouped by cell, each cell's taps in ascending 8 r + t (the order
        // in which R^T r adds them one after another)
        std::vector<int> ord(pi.size());
        for (size_t q = 0; q < ord.size(); ++q) ord[q] = (int)q;
        std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return pi[x] < pi[y]; });
        std::vector<long long> cells;
        std::vector<int> start;
        for (size_t e = 0; e < ord.size(); ++e)
            if (e == 0 || pi[ord[e]] != pi[ord[e - 1]]) {
                cells.push_back(pi[ord[e]]);
                start.push_back((int)e);
            }
        start.push_back((int)ord.size());
        void* tc = nullptr;
        void* tsb = nullptr;
        void* to = nullptr;
        void* tpl = nullptr;
        std::vector<int> plane(h->g.nx + 1);
        for (int i = 0; i <= h->g.nx; ++i)
            plane[i] = (int)(std::lower_bound(cells.begin(), cells.end(), i * h->g.plane) - cells.begin());
        rc = dalloc(h, &tc, cells.size() * sizeof(long long));
        if (!rc) rc = dalloc(h, &tsb, start.size() * sizeof(int));
        if (!rc) rc = dalloc(h, &to, ord.size() * sizeof(int));
        if (!rc) rc = dalloc(h, &tpl, plane.size() * sizeof(int));
        if (rc) return rc;
        h->tap_plane = (int*)tpl;
        h->tap_cell = (long long*)tc;
        h->tap_start = (int*)tsb;
        h->tap_ord = (int*)to;
        h->n_tap_cells = (int)cells.size();
        ACK(cudaMemcpyAsync(h->tap_cell, cells.data(), cells.size() * sizeof(long long), cudaMemcpyHostToDevice,
                            h->stream));
        ACK(cudaMemcpyAsync(h->tap_start, start.data(), start.size() * sizeof(int), cudaMemcpyHostToDevice,
                            h->stream));
        ACK(cudaMemcpyAsync(h->tap_plane, plane.data(), plane.size() * sizeof(int), cudaMemcpyHostToDevice, h->stream));
        ACK(cudaMemcpyAsync(h->tap_ord, ord.data(), ord.size() * sizeof(int), cudaMemcpyHostToDevice, h->stream));
        ACK(cudaStreamSynchronize(h->stream));
    }
    h->n_rec = n_rec;
    h->trace_cap = max_steps;
    return FDTD_OK;
}

int fdtd_b200_adj_forward(FdtdB200Adj* h, int n_steps, int keep_checkpoints, double* traces_out)
{
    if (!h) return FDTD_ERR_NULL;
    if (n_steps < 1 || n_steps > h->trace_cap) return FDTD_ERR_DIM;
    ACK(cudaSetDevice(h->device));
    const int keep = keep_checkpoints ? 1 : 0;
    int rc = keep ? ensure_checkpoints(h, n_steps) : FDTD_OK;
    if (rc) return rc;
    rc = run_sweep(h, h->fwd[keep], n_steps, [&](FdtdB200Adj* s) {
        return s->dbl ? forward_impl<double>(s, n_steps, keep) : forward_impl<float>(s, n_steps, keep);
    });
    if (rc) return rc;
    h->fwd_steps = keep ? n_steps : -1;
    if (traces_out && h->n_rec > 0) {
        const size_t n = (size_t)n_steps * h->n_rec;
        std::vector<unsigned char> buf(n * h->eb);
        ACK(cudaMemcpyAsync(buf.data(), h->traces, buf.size(), cudaMemcpyDeviceToHost, h->stream));
        ACK(cudaStreamSynchronize(h->stream));
        for (size_t q = 0; q < n; ++q) {
            if (h->dbl) memcpy(&traces_out[q], &buf[q * 8], 8);
            else { float f; memcpy(&f, &buf[q * 4], 4); traces_out[q] = f; }
        }
    } else {
        ACK(cudaStreamSynchronize(h->stream));
    }
    return FDTD_OK;
}

int fdtd_b200_adj_backward(FdtdB200Adj* h, const double* dloss_dtrace, double* grad_out)
{
    if (!h || !grad_out || (h->n_rec > 0 && !dloss_dtrace)) return FDTD_ERR_NULL;
    if (h->fwd_steps < 1) return FDTD_ERR_ARG;    // needs a checkpointed forward of the current inputs
    ACK(cudaSetDevice(h->device));
    int rc = ensure_slots(h);
    if (rc) return rc;
    const size_t n = (size_t)h->fwd_steps * h->n_rec;
    if (n > 0) {
        std::vector<unsigned char> buf(n * h->eb);
        for (size_t q = 0; q < n; ++q) {
            if (h->dbl) memcpy(&buf[q * 8], &dloss_dtrace[q], 8);
            else { const float f = (float)dloss_dtrace[q]; memcpy(&buf[q * 4], &f, 4); }
        }
        ACK(cudaMemcpyAsync(h->resid, buf.data(), buf.size(), cudaMemcpyHostToDevice, h->stream));
        ACK(cudaStreamSynchronize(h->stream));
    }
    rc = run_sweep(h, h->bwd, h->fwd_steps, [](FdtdB200Adj* s) {
        return s->dbl ? backward_impl<double>(s) : backward_impl<float>(s);
    });
    if (rc) return rc;
    k_store_grad<<<cell_grid(h->g), kBlock, 0, h->stream>>>(h->g, h->grad, h->grad_ref);
    ACK(cudaGetLastError());
    ACK(cudaMemcpyAsync(grad_out, h->grad_ref, (size_t)h->N * sizeof(double), cudaMemcpyDefault, h->stream));
    ACK(cudaStreamSynchronize(h->stream));
    return FDTD_OK;
}

}  // extern "C"
