/*
 * fdtd_general.cu — two-pass step kernels for arbitrary scenes, plus the
 * small kernels around the step (plate, deposits, samplers, stability check).
 *
 * The two-pass step handles everything the reference's pressure_step does
 * (csrc/kernels/acoustic_fdtd.cpp:1081-1241): rigid walls, cut-cell face
 * fractions, closed faces and the moving-plate faces.  It costs one extra
 * read of P and V compared with the fused single pass (fdtd_fused.cu), which
 * open rooms use.  Memory bound: velocity pass 28 B/cell, pressure pass
 * 20 B/cell (+ fractions and solid mask when present).
 */
#include "fdtd_internal.h"
#include "launch.h"

#include <math.h>

#include <algorithm>

namespace fdtd {

namespace {

__device__ __forceinline__ float4 ld4(const float* p, long long i) { return *reinterpret_cast<const float4*>(p + i); }
__device__ __forceinline__ void st4(float* p, long long i, const float (&v)[4])
{
    *reinterpret_cast<float4*>(p + i) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void unpack(const float4& x, float (&v)[4]) { v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; }

// sum_t w[t] * f[id[t]] in tap order; from_zero starts the running sum at 0.0f
// (the direct samplers, acoustic_fdtd.cpp:1380-1389), otherwise at the first
// product (the precomputed samplers, :1673-1674).  T = the number of taps, known
// for the usual 8 and 4 so that their loads do not wait for one another; 0 = any.
template <int T>
__device__ __forceinline__ float weighted_sum(const float* __restrict__ f, const long long* __restrict__ id,
                                              const float* __restrict__ w, int taps, int from_zero)
{
    float s = 0.0f;
    if constexpr (T > 0) {
        float v[T];
#pragma unroll
        for (int t = 0; t < T; ++t) v[t] = fmul(w[t], f[id[t]]);
        s = from_zero ? fadd(0.0f, v[0]) : v[0];
#pragma unroll
        for (int t = 1; t < T; ++t) s = fadd(s, v[t]);
    } else {
        for (int t = 0; t < taps; ++t) {
            const float v = fmul(w[t], f[id[t]]);
            s = (t == 0 && !from_zero) ? v : fadd(s, v);
        }
    }
    return s;
}

// Threads own four consecutive cells k0 .. k0+3 of a row (k0 a multiple of 4;
// rows start on 8-float boundaries, so every float4 access is aligned).  The
// (row, group) pairs of a plane are numbered consecutively over 1-D blocks,
// so no lane idles when Nz/4 is not a multiple of the warp width (Nz = 74:
// 19 groups per row), and consecutive lanes read consecutive 16-byte groups.
//
// Blocks of 128 threads, six to an SM (80 registers): a small scene is a few
// waves of blocks, and 256-thread blocks, three to an SM, end in a longer tail.
// 170x140x74 scene, whole step: 256 threads 31.8 us, 128 threads 24.8 (64 or 96
// threads 24.9; five or seven 128-thread blocks 26.5 and 25.6); 160x128x128: 42.1
// and 32.7.
constexpr int kCellThreads = 128;
#define GEN_INDEX                                                          \
    const int nq_ = (g.nz + 3) >> 2;                                       \
    const int t_ = blockIdx.x * blockDim.x + threadIdx.x;                  \
    if (t_ >= g.ny * nq_) return;                                          \
    const int j = t_ / nq_;                                                \
    const int k0 = 4 * (t_ - j * nq_);                                     \
    const int i = blockIdx.y;                                              \
    const long long id = ((long long)i * g.ny + j) * g.sz + k0;

// Velocity update on the three staggered face sets (acoustic_fdtd.cpp:1099-1148),
// then closed faces (fraction == 0) are zeroed (:1152-1154).  A thread handles
// Vx(i+1/2,j,k), Vy(i,j+1/2,k) and Vz(i,j,k+1/2) of its four cells where they
// exist; faces that do not exist (and the row padding) keep their stored zero.
// OPEN: a room without walls or plate, with the step's extras (StepExtras).
template <bool OPEN>
__global__ void __launch_bounds__(kCellThreads, 6) k_velocity_general(
    Grid g, Coef cf, Tables tb, const float* __restrict__ p, float* __restrict__ vx,
    float* __restrict__ vy, float* __restrict__ vz, const float* __restrict__ fx,
    const float* __restrict__ fy, const float* __restrict__ fz, const uint8_t* __restrict__ walls,
    const unsigned* __restrict__ gate, PlateFaces pf, StepExtras ex)
{
    // With a plate the kernel before this one is the plate update, which writes no
    // field: the loads start beside it and only the results wait for it.
    if (OPEN || !pf.code) wait_previous();
    release_next();
    if constexpr (OPEN)
        for (int r = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; r < ex.n_rec;
             r += gridDim.x * gridDim.y * blockDim.x)
            ex.row[r] = weighted_sum<8>(p, ex.idx + 8LL * r, ex.w + 8LL * r, 8, 0);
    GEN_INDEX
    // Every load first, from addresses kept inside the field (what a 2nd-order
    // face does not read is loaded and not used): the pass is bound by the latency
    // of L2, and a thread that loads axis by axis keeps fewer in flight
    // (170x140x74 scene, whole step: 35.3 us axis by axis, 34.0 us this way).
    const long long xm = i > 0 ? id - g.plane : id, xp = i < g.nx - 1 ? id + g.plane : id;
    const long long xq = i < g.nx - 2 ? id + 2 * g.plane : id;
    const long long ym = j > 0 ? id - g.sz : id, yp = j < g.ny - 1 ? id + g.sz : id, yq = j < g.ny - 2 ? id + 2 * g.sz : id;
    const unsigned wall = !OPEN && walls ? walls[id >> 2] : 0u;
    float4 p_c = ld4(p, id), p_xm = ld4(p, xm), p_xp = ld4(p, xp), p_xq = ld4(p, xq);
    float4 p_ym = ld4(p, ym), p_yp = ld4(p, yp), p_yq = ld4(p, yq);
    float p_zm = k0 > 0 ? p[id - 1] : 0.0f;
    float2 p_zp = k0 + 4 < g.nz ? *reinterpret_cast<const float2*>(p + id + 4) : make_float2(0.f, 0.f);
    const float4 v_x = ld4(vx, id), v_y = ld4(vy, id), v_z = ld4(vz, id);
    const float ay = __ldg(tb.ay + j), axi = __ldg(tb.ax + i);
    const float axr = __ldg(tb.ax + min(i + 1, g.nx - 1)), ayr = __ldg(tb.ay + min(j + 1, g.ny - 1));
    float az[5], ac[4];
#pragma unroll
    for (int q = 0; q < 5; ++q) az[q] = __ldg(tb.az + min(k0 + q, g.nz - 1));
    float4 f_x = make_float4(1.f, 1.f, 1.f, 1.f), f_y = f_x, f_z = f_x;
    if (wall & kWallX) f_x = ld4(fx, id);
    if (wall & kWallY) f_y = ld4(fy, id);
    if (wall & kWallZ) f_z = ld4(fz, id);
    if constexpr (OPEN) {
        // the source cell is within two cells of this group: every value read there
        // takes the step's sample
        if (ex.cell >= 0 && ex.cell >= id - 2 * g.plane && ex.cell < id + 2 * g.plane + 4) {
            const float sv = *ex.sig;
            if (sv != 0.0f) {
                auto add = [&](float4& v, long long at) {
                    const long long d = ex.cell - at;
                    if (d == 0) v.x = fadd(v.x, sv);
                    if (d == 1) v.y = fadd(v.y, sv);
                    if (d == 2) v.z = fadd(v.z, sv);
                    if (d == 3) v.w = fadd(v.w, sv);
                };
                add(p_c, id); add(p_xm, xm); add(p_xp, xp); add(p_xq, xq);
                add(p_ym, ym); add(p_yp, yp); add(p_yq, yq);
                if (ex.cell == id - 1) p_zm = fadd(p_zm, sv);
                if (ex.cell == id + 4) p_zp.x = fadd(p_zp.x, sv);
                if (ex.cell == id + 5) p_zp.y = fadd(p_zp.y, sv);
            }
        }
    }
    if (!OPEN && pf.code) wait_previous();
    if (!OPEN && gate && gate[kStatusPlate] != 0xFFFFFFFFu) return;   // this step's plate update failed
    if (!OPEN && pf.m > 0 && i == 0 && blockIdx.x == 0)               // the consumed plate forces
        for (int q = threadIdx.x; q < pf.m; q += min((int)blockDim.x, g.ny * nq_)) pf.ext[pf.pack[q].x] = 0.0f;
    float pc[4];
    unpack(p_c, pc);
#pragma unroll
    for (int q = 0; q < 4; ++q) ac[q] = fmaxf(fmaxf(axi, ay), az[q]);
    auto grad = [&](float m, float c, float r, float s, bool fourth) {
        const float d = fsub(r, c), w = fadd(fmul(cf.c1, d), fmul(cf.c2, fsub(s, m)));
        return fourth ? w : d;
    };
    auto face = [&](float v, float gr, float aL, float aR, float fr) {
        const float nv = fmul(fsub(v, fmul(cf.vc, gr)), face_damp(aL, aR, cf.dt));
        return fr == 0.0f ? 0.0f : nv;
    };
    if (i < g.nx - 1) {
        const bool fourth = i > 0 && i < g.nx - 2;
        float pr[4], pm[4], p2[4], v[4], fr[4];
        unpack(p_xp, pr); unpack(p_xm, pm); unpack(p_xq, p2); unpack(v_x, v); unpack(f_x, fr);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float nv = face(v[q], grad(pm[q], pc[q], pr[q], p2[q], fourth), ac[q], fmaxf(fmaxf(axr, ay), az[q]), fr[q]);
            if (k0 + q < g.nz) v[q] = nv;
        }
        st4(vx, id, v);
    }
    if (j < g.ny - 1) {
        const bool fourth = j > 0 && j < g.ny - 2;
        float pr[4], pm[4], p2[4], v[4], fr[4];
        unpack(p_yp, pr); unpack(p_ym, pm); unpack(p_yq, p2); unpack(v_y, v); unpack(f_y, fr);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float nv = face(v[q], grad(pm[q], pc[q], pr[q], p2[q], fourth), ac[q], fmaxf(fmaxf(axi, ayr), az[q]), fr[q]);
            if (k0 + q < g.nz) v[q] = nv;
        }
        st4(vy, id, v);
    }
    {
        const float e[7] = {p_zm, pc[0], pc[1], pc[2], pc[3], p_zp.x, p_zp.y};   // P at k0-1 .. k0+5
        float v[4], fr[4];
        unpack(v_z, v); unpack(f_z, fr);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = k0 + q;
            const float nv = face(v[q], grad(e[q], e[q + 1], e[q + 2], e[q + 3], k > 0 && k < g.nz - 2), ac[q],
                                  fmaxf(fmaxf(axi, ay), az[q + 1]), fr[q]);
            if (k < g.nz - 1) v[q] = nv;
        }
        if (!OPEN && pf.code && k0 <= pf.iz && pf.iz - 1 <= k0 + 3) {   // the plate's faces
            const int node = j + g.ny * i;
            const unsigned c = pf.code[node];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = k0 + q;
                if ((k == pf.iz - 1 && (c & 1u)) || (k == pf.iz && (c & 2u)))
                    v[q] = fmul(fsub(pf.w[node], pf.wp[node]), pf.inv_dt);
            }
        }
        st4(vz, id, v);
    }
}

// Pressure update from the 4th-order divergence (acoustic_fdtd.cpp:894-952,
// :1176-1234).  Faces outside the grid read as zero; with fractions each face
// is scaled by its open fraction; solid cells are skipped (they stay zero in
// both pressure buffers, so the thread writes zero there).  Every load first, as
// in the velocity pass; the fractions of a group near walls come after them.
template <bool OPEN>
__global__ void __launch_bounds__(kCellThreads, 6) k_pressure_general(
    Grid g, Coef cf, Tables tb, const float* __restrict__ p, float* __restrict__ pn,
    const float* __restrict__ vx, const float* __restrict__ vy, const float* __restrict__ vz,
    const float* __restrict__ fx, const float* __restrict__ fy, const float* __restrict__ fz,
    const uint8_t* __restrict__ solid, const uint8_t* __restrict__ walls, const unsigned* __restrict__ gate,
    SubstepOut so, StepExtras ex)
{
    wait_previous();
    release_next();
    if (!OPEN && so.status) {   // what the host waits for, straight into its memory
        const int n_thr = gridDim.x * gridDim.y * blockDim.x;
        const int t = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
        for (int r = t; r < so.n; r += n_thr) so.out[r] = weighted_sum<4>(so.w, so.idx + 4LL * r, so.sw + 4LL * r, 4, 0);
        if (t < kStatusWords) so.h_status[t] = so.status[t];
    }
    GEN_INDEX
    if (!OPEN && gate && gate[kStatusPlate] != 0xFFFFFFFFu) return;   // this step's plate update failed
    const long long P = g.plane, S = g.sz;
    // faces outside the grid: the address stays inside, the value is zero
    const bool x0 = i < g.nx - 1, y0 = j < g.ny - 1;
    const bool x1 = i > 0, x2 = i > 1, x3 = i < g.nx - 2, y1 = j > 0, y2 = j > 1, y3 = j < g.ny - 2;
    const long long ixm = x1 ? id - P : id, ixmm = x2 ? id - 2 * P : id, ixpp = x3 ? id + P : id;
    const long long iym = y1 ? id - S : id, iymm = y2 ? id - 2 * S : id, iypp = y3 ? id + S : id;
    const unsigned wall = !OPEN && walls ? walls[id >> 2] : 0u;
    const float4 q_xp = ld4(vx, id), q_xm = ld4(vx, ixm), q_xpp = ld4(vx, ixpp), q_xmm = ld4(vx, ixmm);
    const float4 q_yp = ld4(vy, id), q_ym = ld4(vy, iym), q_ypp = ld4(vy, iypp), q_ymm = ld4(vy, iymm);
    const float4 q_z = ld4(vz, id);
    const float2 q_zm = k0 >= 2 ? *reinterpret_cast<const float2*>(vz + id - 2) : make_float2(0.f, 0.f);
    const float q_zp = k0 + 4 < g.nz ? vz[id + 4] : 0.0f;
    const float4 q_p = ld4(p, id);
    const float pxy = fminf(__ldg(tb.px + i), __ldg(tb.py + j));
    float pz[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) pz[q] = __ldg(tb.pz + min(k0 + q, g.nz - 1));
    float xp[4], xm[4], xpp[4], xmm[4], yp[4], ym[4], ypp[4], ymm[4], pc[4], out[4];
    float e[7] = {q_zm.x, q_zm.y, q_z.x, q_z.y, q_z.z, q_z.w, q_zp};   // Vz at k0-2 .. k0+4
    unpack(q_xp, xp); unpack(q_xm, xm); unpack(q_xpp, xpp); unpack(q_xmm, xmm);
    unpack(q_yp, yp); unpack(q_ym, ym); unpack(q_ypp, ypp); unpack(q_ymm, ymm);
    unpack(q_p, pc);
    if (OPEN && ex.cell >= id && ex.cell < id + 4) {
        const float sv = *ex.sig;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (ex.cell == id + q && sv != 0.0f) pc[q] = fadd(pc[q], sv);
    }
    uint32_t sol = 0;
    if (wall & kWallNear) {   // elsewhere every fraction is 1
        auto scale = [&](float (&v)[4], const float* f, long long at) {
            float fr[4];
            unpack(ld4(f, at), fr);
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = fmul(v[q], fr[q]);
        };
        if (fx) {
            scale(xp, fx, id); scale(xm, fx, ixm); scale(xpp, fx, ixpp); scale(xmm, fx, ixmm);
        }
        if (fy) {
            scale(yp, fy, id); scale(ym, fy, iym); scale(ypp, fy, iypp); scale(ymm, fy, iymm);
        }
        if (fz) {
#pragma unroll
            for (int q = 0; q < 7; ++q)
                if (k0 + q - 2 >= 0 && k0 + q - 2 < g.nz) e[q] = fmul(e[q], fz[id + q - 2]);
        }
        if (solid) sol = *reinterpret_cast<const uint32_t*>(solid + id);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = k0 + q;
        const float a0 = x0 ? xp[q] : 0.0f, b0 = y0 ? yp[q] : 0.0f;
        const float a1 = x1 ? xm[q] : 0.0f, a2 = x2 ? xmm[q] : 0.0f, a3 = x3 ? xpp[q] : 0.0f;
        const float b1 = y1 ? ym[q] : 0.0f, b2 = y2 ? ymm[q] : 0.0f, b3 = y3 ? ypp[q] : 0.0f;
        const float zp = (k < g.nz - 1) ? e[q + 2] : 0.0f;
        const float zpp = (k < g.nz - 2) ? e[q + 3] : 0.0f;
        const float d1 = fadd(fadd(fsub(a0, a1), fsub(b0, b1)), fsub(zp, e[q + 1]));
        const float d2 = fadd(fadd(fsub(a3, a2), fsub(b3, b2)), fsub(zpp, e[q]));
        const float dv = fadd(fmul(cf.c1, d1), fmul(cf.c2, d2));
        out[q] = fmul(fsub(pc[q], fmul(cf.bulk, dv)), fminf(pxy, pz[q]));
        if (k >= g.nz || ((sol >> (8 * q)) & 0xFFu)) out[q] = 0.0f;
    }
    st4(pn, id, out);
}

// WallCode bytes: the group's own faces and cells, then (after a launch boundary)
// what its pressure update reads around it.  One dimension of blocks over all
// groups, the rows' padding included (code 0): any extent of a room.
#define WALL_INDEX                                                         \
    const long long id = 4 * (blockIdx.x * 256LL + threadIdx.x);           \
    if (id >= g.cells) return;                                             \
    const int i = (int)(id / g.plane), r_ = (int)(id - i * g.plane);       \
    const int j = r_ / g.sz, k0 = r_ - j * g.sz;
__global__ void __launch_bounds__(256) k_wall_own(Grid g, const float* __restrict__ fx, const float* __restrict__ fy,
                                                  const float* __restrict__ fz, const uint8_t* __restrict__ solid,
                                                  uint8_t* __restrict__ code)
{
    WALL_INDEX
    unsigned c = 0;
    for (int q = 0; q < 4; ++q) {
        const int k = k0 + q;
        if (k >= g.nz) break;
        if (fx && i < g.nx - 1 && fx[id + q] != 1.0f) c |= kWallX;
        if (fy && j < g.ny - 1 && fy[id + q] != 1.0f) c |= kWallY;
        if (fz && k < g.nz - 1 && fz[id + q] != 1.0f) c |= kWallZ;
        if (solid && solid[id + q]) c |= kWallSolid;
    }
    code[id >> 2] = (uint8_t)c;
}
__global__ void __launch_bounds__(256) k_wall_near(Grid g, uint8_t* code)
{
    WALL_INDEX
    if (k0 >= g.nz) return;
    unsigned c = code[id >> 2], near = c & (kWallX | kWallY | kWallZ | kWallSolid);
    for (int d = -2; d <= 1; ++d) {
        if (i + d >= 0 && i + d < g.nx) near |= code[(id + d * g.plane) >> 2] & kWallX;
        if (j + d >= 0 && j + d < g.ny) near |= code[(id + (long long)d * g.sz) >> 2] & kWallY;
    }
    if (k0 >= 4) near |= code[(id - 4) >> 2] & kWallZ;
    if (k0 + 4 < g.nz) near |= code[(id + 4) >> 2] & kWallZ;
    if (near) code[id >> 2] = (uint8_t)(c | kWallNear);   // the bits the neighbours read do not change
}

// New displacement of active node q (acoustic_fdtd.cpp:984-1053).
__device__ __forceinline__ float plate_node(int q, int pidx, const int* __restrict__ nb13, float pa, float pb,
                                            const float* __restrict__ w, const float* __restrict__ wp, float fb,
                                            const PlateCoef& pc)
{
    const float W13[13] = {20.f, -8.f, -8.f, -8.f, -8.f, 2.f, 2.f, 2.f, 2.f, 1.f, 1.f, 1.f, 1.f};
    const int* nb = nb13 + 13 * q;
    float bh = 0.0f, bhp = 0.0f;
    for (int t = 0; t < 13; ++t) bh = fadd(bh, fmul(W13[t], w[nb[t]]));
    for (int t = 0; t < 13; ++t) bhp = fadd(bhp, fmul(W13[t], wp[nb[t]]));
    const float vel = fsub(w[pidx], wp[pidx]);
    float wn = fadd(w[pidx], fmul(pc.vd, vel));
    wn = fadd(wn, fmul(pc.a, fadd(fsub(pb, pa), fb)));
    wn = fsub(wn, fmul(pc.bh, bh));
    return fsub(wn, fmul(pc.bk, fsub(bh, bhp)));
}
__device__ __forceinline__ bool plate_bad(float wn) { return !isfinite(wn) || fabsf(wn) > 0.02f; }

// Kirchhoff plate step, one thread per active node.  A node whose new
// displacement is non-finite or above 0.02 m records its ordinal in
// status[kStatusPlate] (the host reports the lowest one) and the step; later
// steps queued behind it then do nothing.
__global__ void k_plate_step(int n_act, const int* __restrict__ act, const int* __restrict__ nb13,
                             const long long* __restrict__ above,
                             const long long* __restrict__ below, const float* __restrict__ w,
                             const float* __restrict__ wp, float* __restrict__ wt,
                             const float* __restrict__ ext, const float* __restrict__ p,
                             PlateCoef pc, unsigned* __restrict__ status, unsigned step)
{
    wait_previous();
    release_next();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_act) return;
    if (*(volatile unsigned*)(status + kStatusPlateStep) < step) return;   // an earlier step of the window failed
    const int pidx = act[q];
    const float wn = plate_node(q, pidx, nb13, above[q] >= 0 ? p[above[q]] : 0.0f, below[q] >= 0 ? p[below[q]] : 0.0f,
                                w, wp, ext[pidx], pc);
    if (plate_bad(wn)) {
        atomicMin(status + kStatusPlate, (unsigned)q);
        atomicMin(status + kStatusPlateStep, step);
    }
    wt[pidx] = wn;
}

// One deposit of the open-cell rule (acoustic_fdtd.cpp:840-872).  The amplitude
// is signal[step] when a signal is given, else `amp`; zero amplitude is a no-op.
__global__ void k_deposit(Deposit d, const float* __restrict__ signal, int step, float amp,
                          float* __restrict__ p)
{
    deposit_apply(d, signal ? signal[step] : amp, p);
}

// out[r] = sum_t w[r*taps+t] * f[idx[r*taps+t]].
__global__ void k_wsum(const float* __restrict__ f, const long long* __restrict__ idx,
                       const float* __restrict__ w, int n_out, int taps, int from_zero,
                       float* __restrict__ out)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_out) return;
    const long long* id = idx + (long long)taps * r;
    const float* ww = w + (long long)taps * r;
    out[r] = taps == 8 ? weighted_sum<8>(f, id, ww, 8, from_zero)
           : taps == 4 ? weighted_sum<4>(f, id, ww, 4, from_zero) : weighted_sum<0>(f, id, ww, taps, from_zero);
}

// Stability check (acoustic_fdtd.cpp:1245-1268): cells phase, phase+1013, ...
// (reference flat order) that are non-finite or beyond +-2e3 Pa record their
// flat index; the latch keeps the first failing step for async stepping.
__global__ void k_check(Grid g, const float* __restrict__ p, long long n_cells, int phase,
                        unsigned* __restrict__ status, int step, const unsigned* __restrict__ gate)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long q = phase + t * kCheckStride;
    if (q >= n_cells) return;
    if (gate && gate[kStatusPlate] != 0xFFFFFFFFu) return;   // this step's plate update failed

    const int k = (int)(q % g.nz);
    const long long ij = q / g.nz;
    const int j = (int)(ij % g.ny);
    const long long i = ij / g.ny;
    const float v = p[(i * g.ny + j) * g.sz + k];
    if (!isfinite(v) || v > 2e3f || v < -2e3f) {
        atomicMin(status + kStatusCell, (unsigned)q);
        atomicCAS(status + kStatusLatch, 0xFFFFFFFFu, (unsigned)step);
    }
}


// Zeroes n floats unless this step's plate update failed (the consumed plate
// forces of a step whose success is only known after it ran).
__global__ void k_zero_gated(float* __restrict__ x, int n, const unsigned* __restrict__ gate)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n || gate[kStatusPlate] != 0xFFFFFFFFu) return;
    x[q] = 0.0f;
}

// What a substep starts with: the pending plate forces, (node, value) pairs in
// host memory, go into the device force buffer (all its other entries are zero),
// and the plate guard is cleared.
__global__ void k_substep_begin(float* __restrict__ ext, const int2* __restrict__ h_pack, int2* __restrict__ pack, int m,
                                unsigned* __restrict__ status)
{
    release_next();
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q == 0) status[kStatusPlate] = status[kStatusPlateStep] = 0xFFFFFFFFu;
    if (q >= m) return;
    const int2 v = h_pack[q];
    pack[q] = v;
    ext[v.x] = __int_as_float(v.y);
}

// One plane of a field across the given axis, rows of the remaining two axes
// in (i, j, k) order: axis 0 -> (Ny, Nz), 1 -> (Nx, Nz), 2 -> (Nx, Ny).
__global__ void k_slice(const float* __restrict__ f, Grid g, int axis, int idx, float* __restrict__ out,
                        int na, int nb)
{
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long long)na * nb) return;
    const long long a = q / nb, b = q % nb;
    const long long off = axis == 0 ? ((long long)idx * g.ny + a) * g.sz + b
                        : axis == 1 ? (a * g.ny + idx) * g.sz + b
                                    : (a * g.ny + b) * g.sz + idx;
    out[q] = f[off];
}
}  // namespace

cudaError_t launch_velocity_general(const Grid& g, const Coef& cf, const Tables& tb,
                                    const float* p, float* vx, float* vy, float* vz,
                                    const float* fx, const float* fy, const float* fz, const uint8_t* walls,
                                    cudaStream_t s, const unsigned* gate, const PlateFaces* pf)
{
    dim3 block(kCellThreads, 1, 1);
    dim3 grid((g.ny * ((g.nz + 3) / 4) + kCellThreads - 1) / kCellThreads, g.nx, 1);
    return launch_after(k_velocity_general<false>, grid, block, 0, s, g, cf, tb, p, vx, vy, vz, fx, fy, fz, walls, gate,
                        pf ? *pf : PlateFaces(), StepExtras());
}

cudaError_t launch_pressure_general(const Grid& g, const Coef& cf, const Tables& tb,
                                    const float* p, float* pn, const float* vx, const float* vy,
                                    const float* vz, const float* fx, const float* fy,
                                    const float* fz, const uint8_t* solid, const uint8_t* walls, cudaStream_t s,
                                    const unsigned* gate, const SubstepOut* so)
{
    dim3 block(kCellThreads, 1, 1);
    dim3 grid((g.ny * ((g.nz + 3) / 4) + kCellThreads - 1) / kCellThreads, g.nx, 1);
    return launch_after(k_pressure_general<false>, grid, block, 0, s, g, cf, tb, p, pn, vx, vy, vz, fx, fy, fz, solid,
                        walls, gate, so ? *so : SubstepOut(), StepExtras());
}

cudaError_t launch_open_step(const Grid& g, const Coef& cf, const Tables& tb, const float* p, float* pn, float* vx,
                             float* vy, float* vz, const StepExtras& ex, cudaStream_t s)
{
    dim3 block(kCellThreads, 1, 1);
    dim3 grid((g.ny * ((g.nz + 3) / 4) + kCellThreads - 1) / kCellThreads, g.nx, 1);
    const float* none = nullptr;
    const uint8_t* no_walls = nullptr;
    const unsigned* no_gate = nullptr;
    const cudaError_t e = launch_after(k_velocity_general<true>, grid, block, 0, s, g, cf, tb, p, vx, vy, vz, none, none,
                                       none, no_walls, no_gate, PlateFaces(), ex);
    if (e != cudaSuccess) return e;
    return launch_after(k_pressure_general<true>, grid, block, 0, s, g, cf, tb, p, pn, (const float*)vx,
                        (const float*)vy, (const float*)vz, none, none, none, no_walls, no_walls, no_gate, SubstepOut(),
                        ex);
}

cudaError_t launch_plate_step(int n_act, const int* act, const int* nb13, const long long* above,
                              const long long* below, const float* w, const float* wp, float* wt,
                              const float* ext, const float* p, const PlateCoef& pc,
                              unsigned* status, unsigned step, cudaStream_t s)
{
    if (n_act <= 0) return cudaSuccess;
    return launch_after(k_plate_step, dim3((n_act + 127) / 128), dim3(128), 0, s, n_act, act, nb13, above, below, w, wp,
                        wt, ext, p, pc, status, step);
}

cudaError_t launch_wall_codes(const Grid& g, const float* fx, const float* fy, const float* fz, const uint8_t* solid,
                              uint8_t* code, cudaStream_t s)
{
    const unsigned grid = (unsigned)((g.cells / 4 + 255) / 256);
    k_wall_own<<<grid, 256, 0, s>>>(g, fx, fy, fz, solid, code);
    k_wall_near<<<grid, 256, 0, s>>>(g, code);
    return cudaGetLastError();
}

cudaError_t launch_deposit(const Deposit& d, const float* signal, int step, float amp, float* p,
                           cudaStream_t s)
{
    k_deposit<<<1, 1, 0, s>>>(d, signal, step, amp, p);
    return cudaGetLastError();
}

cudaError_t launch_wsum(const float* f, const long long* idx, const float* w, int n_out, int taps,
                        int from_zero, float* out, cudaStream_t s)
{
    if (n_out <= 0) return cudaSuccess;
    k_wsum<<<(n_out + 127) / 128, 128, 0, s>>>(f, idx, w, n_out, taps, from_zero, out);
    return cudaGetLastError();
}

cudaError_t launch_check(const Grid& g, const float* p, long long n_cells, int phase,
                         unsigned* status, int step, cudaStream_t s, const unsigned* gate)
{
    if (phase >= n_cells) return cudaSuccess;
    const long long n = (n_cells - phase + kCheckStride - 1) / kCheckStride;
    const int blocks = (int)((n + 255) / 256);
    k_check<<<blocks, 256, 0, s>>>(g, p, n_cells, phase, status, step, gate);
    return cudaGetLastError();
}

cudaError_t launch_zero_gated(float* x, int n, const unsigned* gate, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    k_zero_gated<<<(n + 255) / 256, 256, 0, s>>>(x, n, gate);
    return cudaGetLastError();
}

cudaError_t launch_substep_begin(float* ext, const int2* h_pack, int2* pack, int m, unsigned* status, cudaStream_t s)
{
    k_substep_begin<<<std::max((m + 127) / 128, 1), 128, 0, s>>>(ext, h_pack, pack, m, status);
    return cudaGetLastError();
}

cudaError_t launch_slice(const float* f, const Grid& g, int axis, int idx, float* out, int na, int nb,
                         cudaStream_t s)
{
    const long long n = (long long)na * nb;
    if (n <= 0) return cudaSuccess;
    k_slice<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(f, g, axis, idx, out, na, nb);
    return cudaGetLastError();
}

}  // namespace fdtd
