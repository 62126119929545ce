/*
 * fdtd_resident.cu — many steps of a small open room in one launch, its fields
 * held on chip.
 *
 * A room of up to about 1.2M cells fits the registers and shared memory of the
 * 148 SMs.  One CTA per SM owns a brick of cells; P, Vx, Vy and Vz of the
 * brick stay on chip from the first step of a call to the last, and the only
 * traffic per step is the bricks' boundary: each CTA hands the three outer
 * layers of its new P to its six neighbours through L2.  Velocities are never
 * exchanged: the faces a brick's divergence needs beyond its own (two below,
 * one above, per axis) are updated by the brick itself from its P halo, with
 * the same operations on the same operands as in the brick that owns them.
 *
 * The step of a small room is bound by latency, not by bytes or operations:
 * as one launch per step the march of fdtd_fused.cu spends 10.8 us on the 64^3
 * room (a launch, then six dependent pipeline iterations for one plane per
 * CTA), where 32 B per cell from L2 take about 1 us and its arithmetic 0.3 us.
 * Measured per step, march / here: 32^3 9.4 / 2.1 us, 64^3 12.2 / 3.55,
 * 109x87x61 17.1 / 5.8, 96^3 22 / 6.5, 128x96x96 25 / 7.9.  What is left is
 * the exchange's round trip through L2 and two barriers (1.5 us) and, from
 * there on, instruction issue (2.3 ns per quad and SM).
 *
 * Exchange: a boundary quad (four cells) travels as four 8-byte words
 * {value, step number}, written and polled with relaxed 64-bit accesses, so
 * a word validates itself and no fence or flag round trip is needed.  Two
 * buffers alternate by step: a CTA overwrites a buffer two steps later, after
 * it has received its neighbours' next step, which they send only when they
 * have read this one.  Step numbers grow over the handle's life, so words of
 * an earlier launch never match.  The launch is cooperative (all CTAs are
 * resident together), and every poll is bounded: a wait that runs out sets
 * the timeout status word and the CTA leaves; the others see the word, or
 * their own bound.
 *
 * Per step and CTA: velocities of own quads (registers) and halo faces (shared
 * memory); barrier; P of own quads, published as it is computed; the
 * neighbours' layers into the P halo; barrier.  A thread owns a quad along k
 * over L consecutive planes.  With L = 1 (rooms up to about 300k cells) its
 * fields and damping factors stay in registers; with more they are read from
 * shared memory and the damping is recomputed, which costs less than spilling:
 * beside 200 KB of shared memory the L1 holds almost none of a spilled frame
 * (with the fields of four planes in registers the 96^3 room took 16.3 us per
 * step, so 7.9).  The rows and quads of a brick are template parameters, so
 * that a stencil's shared-memory accesses are one base and constant offsets.
 *
 * Arithmetic is that of fdtd_fused.cu's general path operation for operation
 * (csrc/kernels/acoustic_fdtd.cpp:1099-1148, :894-952, :1176-1234): results
 * are the step-at-a-time kernels' bit for bit.
 */
#include "fdtd_internal.h"
#include "fdtd_tma.h"

#include <algorithm>
#include <atomic>
#include <type_traits>

namespace fdtd {

namespace {

constexpr int kResThreads = 512;       // threads of a CTA
constexpr int kResRecords = 4;         // exchange records a thread receives per step, at most
constexpr int kResQuads = 2;           // halo quads of x and y faces a thread updates, at most
constexpr int kResScalars = 2;         // halo z faces a thread updates, at most
constexpr int kResMaxTaps = 1024;      // most receiver taps the kernel records
constexpr int kResSmem = 226 * 1024;

// Bank conflicts of 16-byte accesses over rows of Q quads at row stride s
// (floats): the most of eight consecutive threads that share a bank group.
constexpr int conflict(int Q, int s)
{
    int worst = 1;
    for (int g0 = 0; g0 < 64; g0 += 8) {
        int hit[8] = {};
        for (int t = g0; t < g0 + 8; ++t) {
            const int b = (t / Q * s / 4 + t % Q) % 8;
            if (++hit[b] > worst) worst = hit[b];
        }
    }
    return worst;
}
constexpr int row_stride(int Q, int least)
{
    int best = least;
    for (int s = least; s < least + 32; s += 4)
        if (conflict(Q, s) < conflict(Q, best)) best = s;
    return best;
}

// The rows and quads of a brick and what follows from them (floats).
template <int Q_, int BJ_>
struct Brick {
    static constexpr int Q = Q_, BJ = BJ_, BK = 4 * Q;
    static constexpr int SP = row_stride(Q, BK + 8);   // rows of P (cells -4 .. BK+3)
    static constexpr int SV = row_stride(Q, BK);       // rows of Vx and Vy
    static constexpr int SZ = row_stride(Q, BK + 8);   // rows of Vz (faces -4 .. BK+3)
    static constexpr int PP = (BJ + 6) * SP;           // planes of P (rows -3 .. BJ+2)
    static constexpr int PX = BJ * SV, PY = (BJ + 3) * SV, PZ = BJ * SZ;
    static constexpr int FX = 3 * BJ * Q;              // records of an x face
};

// Shared-memory map of a brick of bi planes (floats): P of planes -3 .. bi+2, Vx
// faces -2 .. bi, Vy rows -2 .. BJ, Vz; alpha of planes -2 .. bi+1, rows -2 ..
// BJ+1 and cells -4 .. BK+3; the pressure damping of planes, rows and cells;
// (cell offset, tap) pairs of the receivers' taps in the brick; per-thread
// descriptors.
struct ResMap {
    int p, vx, vy, vz, ax, ay, az, px, py, pz, taps, desc, total;
};

struct ResArgs {
    Grid g;
    Coef cf;
    Tables tb;
    const float* p;
    float* pn;
    const float* vin[3];
    float* vout[3];
    unsigned* status;
    unsigned wait_us;
    int hold_brick;                    // publishes nothing (-1: none)
    int L, bi;                         // planes per thread, planes of a brick
    int nbi, nbj, nbk;                 // bricks
    ResMap m;
    uint4* xbuf;                       // exchange: 32-byte records [parity][brick][record]
    unsigned epoch;                    // step s of this launch carries epoch + s + 1
    int steps;
    // point source: sig[step0 + s] goes into (si, sj, sk) before step s, dep_from <= s < dep_to
    const float* sig;
    int step0, dep_from, dep_to, si, sj, sk;
    // receivers' taps: padded index of tap t; tap_out[s * n_taps + t] = P after step s
    const long long* tap_idx;
    int n_taps, rec_steps;
    float* tap_out;
};

__device__ __forceinline__ void put4(float* p, const float (&v)[4])
{
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void get4(const float* p, float (&v)[4])
{
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}

// One record, published when `on` (predicated: a branch per face would cost
// more than the stores).
__device__ __forceinline__ void post4(bool on, uint4* dst, const float (&v)[4], unsigned tag)
{
    asm volatile(
        "{\n .reg .pred q;\n .reg .b64 a, b, c, d;\n setp.ne.u32 q, %0, 0;\n"
        " mov.b64 a, {%2, %6};\n mov.b64 b, {%3, %6};\n mov.b64 c, {%4, %6};\n mov.b64 d, {%5, %6};\n"
        " @q st.relaxed.gpu.global.v2.b64 [%1], {a, b};\n @q st.relaxed.gpu.global.v2.b64 [%1+16], {c, d};\n}\n"
        ::"r"((unsigned)on), "l"(dst), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])),
          "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])), "r"(tag) : "memory");
}
// One record's 32 bytes as read now; landed() says whether they carry `tag`.
struct Record {
    unsigned v[4], t[4];
    __device__ __forceinline__ void load(bool on, const uint4* src)
    {
        asm volatile(
            "{\n .reg .pred q;\n .reg .b64 a, b, c, d;\n setp.ne.u32 q, %8, 0;\n"
            " mov.b64 a, 0;\n mov.b64 b, 0;\n mov.b64 c, 0;\n mov.b64 d, 0;\n"
            " @q ld.relaxed.gpu.global.v2.b64 {a, b}, [%9];\n @q ld.relaxed.gpu.global.v2.b64 {c, d}, [%9+16];\n"
            " mov.b64 {%0, %4}, a;\n mov.b64 {%1, %5}, b;\n mov.b64 {%2, %6}, c;\n mov.b64 {%3, %7}, d;\n}\n"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3])
            : "r"((unsigned)on), "l"(src) : "memory");
    }
    __device__ __forceinline__ bool landed(unsigned tag) const
    {
        return ((t[0] ^ tag) | (t[1] ^ tag) | (t[2] ^ tag) | (t[3] ^ tag)) == 0u;
    }
    __device__ __forceinline__ void store(bool on, float* dst) const
    {
        asm volatile(
            "{\n .reg .pred q;\n setp.ne.u32 q, %0, 0;\n @q st.shared.v4.b32 [%1], {%2, %3, %4, %5};\n}\n"
            ::"r"((unsigned)on), "r"(smem_u32(dst)), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
    }
};

// Gradient of one face: 4th order, or 2nd next to the grid's ends (selected, not
// branched on: the branch took 0.9 of 4.3 us per step on the 64^3 room).
__device__ __forceinline__ float res_grad(const Coef& cf, float pm, float p0, float p1, float p2, bool fourth)
{
    const float d = fsub(p1, p0), w = fadd(fmul(cf.c1, d), fmul(cf.c2, fsub(p2, pm)));
    return fourth ? w : d;
}
__device__ __forceinline__ float res_vel(const Coef& cf, float v, float grad, float damp)
{
    return fmul(fsub(v, fmul(cf.vc, grad)), damp);
}

template <bool KEEP, class B>
__global__ void __launch_bounds__(kResThreads, 1) k_resident(const __grid_constant__ ResArgs a)
{
    constexpr int Q = B::Q, BJ = B::BJ, BK = B::BK, SP = B::SP, SV = B::SV, SZ = B::SZ;
    constexpr int PP = B::PP, PX = B::PX, PY = B::PY, PZ = B::PZ, FX = B::FX, NT = kResThreads;
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_ntap;
    __shared__ float s_pre;            // the source cell's pressure before its next sample
    const Grid g = a.g;
    const Coef cf = a.cf;
    const ResMap m = a.m;
    const int tid = threadIdx.x, b = blockIdx.x;
    const int bz = b % a.nbk, by = (b / a.nbk) % a.nbj, bx = b / (a.nbk * a.nbj);
    const int L = KEEP ? 1 : a.L, bi = a.bi;
    const int i0 = bx * bi, j0 = by * BJ, k0 = bz * BK;
    const int FY = 3 * bi * Q, FZ = bi * BJ;           // records of a y and of a z face
    // offsets of cell / face (0, 0, 0) in sm
    const int Ps = m.p + 3 * PP + 3 * SP + 4, Xs = m.vx + 2 * PX, Ys = m.vy + 2 * SV, Zs = m.vz + 4;
    float* const axs = sm + m.ax + 2;
    float* const ays = sm + m.ay + 2;
    float* const azs = sm + m.az + 4;
    float* const pxs = sm + m.px;
    float* const pys = sm + m.py;
    float* const pzs = sm + m.pz;
    int2* const taps = reinterpret_cast<int2*>(sm + m.taps);

    for (int e = 4 * tid; e < m.total; e += 4 * NT) *reinterpret_cast<float4*>(sm + e) = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid == 0) { s_ntap = 0; s_pre = 0.0f; }
    __syncthreads();
    for (int e = tid - 2; e < bi + 2; e += NT) axs[e] = (i0 + e >= 0 && i0 + e < g.nx) ? __ldg(a.tb.ax + i0 + e) : 0.0f;
    for (int e = tid - 2; e < BJ + 2; e += NT) ays[e] = (j0 + e >= 0 && j0 + e < g.ny) ? __ldg(a.tb.ay + j0 + e) : 0.0f;
    for (int e = tid - 4; e < BK + 4; e += NT) azs[e] = (k0 + e >= 0 && k0 + e < g.nz) ? __ldg(a.tb.az + k0 + e) : 0.0f;
    for (int e = tid; e < bi; e += NT) pxs[e] = (i0 + e < g.nx) ? __ldg(a.tb.px + i0 + e) : 1.0f;
    for (int e = tid; e < BJ; e += NT) pys[e] = (j0 + e < g.ny) ? __ldg(a.tb.py + j0 + e) : 1.0f;
    for (int e = tid; e < BK; e += NT) pzs[e] = (k0 + e < g.nz) ? __ldg(a.tb.pz + k0 + e) : 1.0f;
    // the source sample of the first step, on every copy of its cell
    const bool dep0 = a.sig && a.dep_from <= 0 && a.dep_to > 0;
    const float amp0 = dep0 ? __ldg(a.sig + a.step0) : 0.0f;
    // P of the brick and of its halo (never the edges and corners of the box)
    for (int e = tid; e < (bi + 6) * (BJ + 6) * (Q + 2); e += NT) {
        const int c = e % (Q + 2) - 1, r = e / (Q + 2) % (BJ + 6) - 3, l = e / ((Q + 2) * (BJ + 6)) - 3;
        const int out = (c < 0 || c >= Q) + (r < 0 || r >= BJ) + (l < 0 || l >= bi);
        const int i = i0 + l, j = j0 + r, k = k0 + 4 * c;
        if (out > 1 || i < 0 || i >= g.nx || j < 0 || j >= g.ny || k < 0 || k >= g.nz) continue;
        float v[4];
        get4(a.p + i * g.plane + (long long)j * g.sz + k, v);
        if (dep0 && amp0 != 0.0f && i == a.si && j == a.sj) {
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (k + t == a.sk) v[t] = fadd(v[t], amp0);
        }
        put4(sm + Ps + l * PP + r * SP + 4 * c, v);
    }
    // halo faces' velocities: x faces -2, -1, bi; y faces -2, -1, BJ; z faces -2, -1, BK
    for (int e = tid; e < FX; e += NT) {
        const int c = e % Q, r = e / Q % BJ, w = e / (Q * BJ), f = w < 2 ? w - 2 : bi;
        const int i = i0 + f, j = j0 + r, k = k0 + 4 * c;
        if (i < 0 || i >= g.nx || j >= g.ny || k >= g.nz) continue;
        float v[4];
        get4(a.vin[0] + i * g.plane + (long long)j * g.sz + k, v);
        put4(sm + Xs + f * PX + r * SV + 4 * c, v);
    }
    for (int e = tid; e < FY; e += NT) {
        const int c = e % Q, w = e / Q % 3, l = e / (3 * Q), f = w < 2 ? w - 2 : BJ;
        const int i = i0 + l, j = j0 + f, k = k0 + 4 * c;
        if (i >= g.nx || j < 0 || j >= g.ny || k >= g.nz) continue;
        float v[4];
        get4(a.vin[1] + i * g.plane + (long long)j * g.sz + k, v);
        put4(sm + Ys + l * PY + f * SV + 4 * c, v);
    }
    for (int e = tid; e < 3 * FZ; e += NT) {
        const int w = e % 3, r = e / 3 % BJ, l = e / (3 * BJ), f = w < 2 ? w - 2 : BK;
        const int i = i0 + l, j = j0 + r, k = k0 + f;
        if (i >= g.nx || j >= g.ny || k < 0 || k >= g.nz) continue;
        sm[Zs + l * PZ + r * SZ + f] = __ldg(a.vin[2] + i * g.plane + (long long)j * g.sz + k);
    }
    for (int t = tid; t < a.n_taps; t += NT) {
        const long long id = a.tap_idx[t];
        const int i = (int)(id / g.plane), rem = (int)(id - i * g.plane);
        const int l = i - i0, r = rem / g.sz - j0, k = rem % g.sz - k0;
        if (l < 0 || l >= bi || r < 0 || r >= BJ || k < 0 || k >= BK) continue;
        const bool src = a.sig && i == a.si && j0 + r == a.sj && k0 + k == a.sk;
        taps[atomicAdd(&s_ntap, 1)] = make_int2(src ? -1 : Ps + l * PP + r * SP + k, t);
    }

    // this thread's quads: cells k0+4q .. +3 of row j, planes l0 .. l0+L-1
    const int qq = tid % Q, lj = tid / Q % BJ, l0 = tid / (Q * BJ) * L;
    const int gj = j0 + lj, gk = k0 + 4 * qq;
    const bool own = l0 < bi && gj < g.ny && gk < g.nz;
    const int nl = own ? max(0, min(min(L, bi - l0), g.nx - i0 - l0)) : 0;   // existing planes
    const long long gid = (long long)(i0 + l0) * g.plane + (long long)gj * g.sz + gk;
    const int pc = Ps + l0 * PP + lj * SP + 4 * qq;
    const int xc = Xs + l0 * PX + lj * SV + 4 * qq;
    const int yc = Ys + l0 * PY + lj * SV + 4 * qq;
    const int zc = Zs + l0 * PZ + lj * SZ + 4 * qq;
    for (int l = 0; l < nl; ++l) {
        float v[4];
        get4(a.vin[0] + gid + l * g.plane, v);
        put4(sm + xc + l * PX, v);
        get4(a.vin[1] + gid + l * g.plane, v);
        put4(sm + yc + l * PY, v);
        get4(a.vin[2] + gid + l * g.plane, v);
        put4(sm + zc + l * PZ, v);
    }
    __syncthreads();
    float P[KEEP ? 4 : 1], VX[KEEP ? 4 : 1], VY[KEEP ? 4 : 1], VZ[KEEP ? 4 : 1];
    float DX[KEEP ? 4 : 1], DY[KEEP ? 4 : 1], DZ[KEEP ? 4 : 1], PD[KEEP ? 4 : 1];
    if constexpr (KEEP) {
        const bool in = nl > 0;
        const float axl = in ? axs[l0] : 0.0f, axr = in ? axs[l0 + 1] : 0.0f;
        const float ay = in ? ays[lj] : 0.0f, ayr = in ? ays[lj + 1] : 0.0f;
        const float pxy = in ? fminf(pxs[l0], pys[lj]) : 1.0f;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            P[t] = in ? sm[pc + t] : 0.0f;
            VX[t] = in ? sm[xc + t] : 0.0f;
            VY[t] = in ? sm[yc + t] : 0.0f;
            VZ[t] = in ? sm[zc + t] : 0.0f;
            const float az = in ? azs[4 * qq + t] : 0.0f, azr = in ? azs[4 * qq + t + 1] : 0.0f;
            const float c = fmaxf(axl, fmaxf(ay, az));
            DX[t] = face_damp(c, fmaxf(axr, fmaxf(ay, az)), cf.dt);
            DY[t] = face_damp(c, fmaxf(axl, fmaxf(ayr, az)), cf.dt);
            DZ[t] = face_damp(c, fmaxf(axl, fmaxf(ay, azr)), cf.dt);
            PD[t] = in ? fminf(pxy, pzs[4 * qq + t]) : 1.0f;
        }
    }

    const bool y4 = gj > 0 && gj < g.ny - 2, yex = gj <= g.ny - 2;
    int z4 = 0, zex = 0, cex = 0;      // own z faces of 4th order, existing; existing cells
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        z4 |= (gk + t > 0 && gk + t < g.nz - 2) ? 1 << t : 0;
        zex |= (gk + t <= g.nz - 2) ? 1 << t : 0;
        cex |= (gk + t < g.nz) ? 1 << t : 0;
    }
    // a warp whose faces and cells all exist, with 4th-order gradients, takes the body without tests
    const bool inner = nl == L && i0 + l0 > 0 && i0 + l0 + L < g.nx - 1 && y4 && yex && z4 == 15 && zex == 15 && cex == 15;
    const bool fast = __all_sync(0xFFFFFFFFu, inner || nl == 0);
    // A brick's records: x faces [3][BJ][Q] low then high, y faces [bi][3][Q],
    // z faces [bi][BJ].  What this thread publishes of plane l0: its place in
    // the low faces, and the faces its row and quad belong to.
    const int rec = 2 * (FX + FY + FZ), nbricks = a.nbi * a.nbj * a.nbk;
    const int rx0 = (l0 * BJ + lj) * Q + qq;
    const int ry0 = 2 * FX + (l0 * 3 + (lj < 3 ? lj : lj - BJ + 3)) * Q + qq;
    const int rz0 = 2 * (FX + FY) + l0 * BJ + lj;
    const unsigned pub = (lj < 3 && by > 0 ? 1u : 0u) | (lj >= BJ - 3 && by + 1 < a.nbj ? 2u : 0u) |
                         (qq == 0 && bz > 0 ? 4u : 0u) | (qq == Q - 1 && bz + 1 < a.nbk ? 8u : 0u);
    const int pxl = bx > 0 ? 3 : 0, pxh = bx + 1 < a.nbi ? bi - 3 : bi;   // planes below / from which x faces are published
    // the source cell, when this thread owns it: its plane and place in the quad
    const bool src_here = a.sig && nl > 0 && gj == a.sj && a.sk >= gk && a.sk < gk + 4 && a.si >= i0 + l0 &&
                          a.si < i0 + l0 + nl;
    const int src_l = src_here ? a.si - i0 - l0 : -1, src_t = a.sk - gk;

    // The halo faces this thread updates each step: quads of x or y faces (quad
    // offsets of P and of the velocity in 16 bits each, damping) and single z
    // faces (offsets in 16 bits each), taken from the other end of the CTA so
    // that the warps share them evenly.  Cells of a ragged quad that do not
    // exist have zero P and velocity around them and feed no cell that exists.
    unsigned hq[kResQuads], hz[kResScalars];
    float hq_d[kResQuads][4], hz_d[kResScalars];
    unsigned hq_on = 0, hq_4 = 0, hq_y = 0, hz_on = 0, hz_4 = 0;
#pragma unroll
    for (int u = 0; u < kResQuads; ++u) {
        const int e = tid + u * NT;
        hq[u] = 0;
#pragma unroll
        for (int t = 0; t < 4; ++t) hq_d[u][t] = 1.0f;
        if (e < FX) {
            const int c = e % Q, r = e / Q % BJ, w = e / (Q * BJ), f = w < 2 ? w - 2 : bi, i = i0 + f;
            if (i < 0 || i > g.nx - 2 || j0 + r >= g.ny || k0 + 4 * c >= g.nz) continue;
            hq[u] = (unsigned)(Ps + f * PP + r * SP + 4 * c) >> 2 | (unsigned)(Xs + f * PX + r * SV + 4 * c) >> 2 << 16;
            hq_on |= 1u << u;
            if (i > 0 && i < g.nx - 2) hq_4 |= 1u << u;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float myz = fmaxf(ays[r], azs[4 * c + t]);
                hq_d[u][t] = face_damp(fmaxf(axs[f], myz), fmaxf(axs[f + 1], myz), cf.dt);
            }
        } else if (e < FX + FY) {
            const int v = e - FX, c = v % Q, w = v / Q % 3, l = v / (3 * Q), f = w < 2 ? w - 2 : BJ, j = j0 + f;
            if (i0 + l >= g.nx || j < 0 || j > g.ny - 2 || k0 + 4 * c >= g.nz) continue;
            hq[u] = (unsigned)(Ps + l * PP + f * SP + 4 * c) >> 2 | (unsigned)(Ys + l * PY + f * SV + 4 * c) >> 2 << 16;
            hq_y |= 1u << u;
            hq_on |= 1u << u;
            if (j > 0 && j < g.ny - 2) hq_4 |= 1u << u;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float az = azs[4 * c + t];
                hq_d[u][t] = face_damp(fmaxf(axs[l], fmaxf(ays[f], az)), fmaxf(axs[l], fmaxf(ays[f + 1], az)), cf.dt);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < kResScalars; ++u) {
        const int e = NT - 1 - tid + u * NT;
        hz[u] = 0;
        hz_d[u] = 1.0f;
        if (e >= 3 * FZ) continue;
        const int w = e % 3, r = e / 3 % BJ, l = e / (3 * BJ), f = w < 2 ? w - 2 : BK, k = k0 + f;
        if (i0 + l >= g.nx || j0 + r >= g.ny || k < 0 || k > g.nz - 2) continue;
        hz[u] = (unsigned)(Ps + l * PP + r * SP + f) | (unsigned)(Zs + l * PZ + r * SZ + f) << 16;
        hz_on |= 1u << u;
        if (k > 0 && k < g.nz - 2) hz_4 |= 1u << u;
        const float mxy = fmaxf(axs[l], ays[r]);
        hz_d[u] = face_damp(fmaxf(mxy, azs[f]), fmaxf(mxy, azs[f + 1]), cf.dt);
    }
    // the records this thread receives each step: their place in a parity's half
    // of the exchange buffer (19 bits) and their quad of the P array (13 bits)
    unsigned r_at[kResRecords], r_mask = 0;
#pragma unroll
    for (int u = 0; u < kResRecords; ++u) {
        const int e = tid + u * NT;
        r_at[u] = 0;
        if (e >= rec) continue;
        int axis, hi, v, step, li, lr, c;      // hi: the next brick's first layers, else the last of the one before
        if (e < 2 * FX) {
            axis = 0; hi = e >= FX; v = e - hi * FX; step = a.nbj * a.nbk;
            c = v % Q; lr = v / Q % BJ; li = v / (Q * BJ) + (hi ? bi : -3);
        } else if (e < 2 * (FX + FY)) {
            const int e1 = e - 2 * FX;
            axis = 1; hi = e1 >= FY; v = e1 - hi * FY; step = a.nbk;
            c = v % Q; lr = v / Q % 3 + (hi ? BJ : -3); li = v / (3 * Q);
        } else {
            const int e1 = e - 2 * (FX + FY);
            axis = 2; hi = e1 >= FZ; v = e1 - hi * FZ; step = 1;
            lr = v % BJ; li = v / BJ; c = hi ? Q : -1;
        }
        const int at = axis == 0 ? bx : axis == 1 ? by : bz, last = (axis == 0 ? a.nbi : axis == 1 ? a.nbj : a.nbk) - 1;
        if (hi ? at == last : at == 0) continue;
        if (i0 + li >= g.nx || j0 + lr >= g.ny || k0 + 4 * c >= g.nz) continue;
        const int first = axis == 0 ? 0 : axis == 1 ? 2 * FX : 2 * (FX + FY), face = axis == 0 ? FX : axis == 1 ? FY : FZ;
        r_at[u] = (unsigned)(rec * (hi ? b + step : b - step) + first + (hi ? 0 : face) + v) << 13 |
                  (unsigned)(Ps - m.p + li * PP + lr * SP + 4 * c) >> 2;
        r_mask |= 1u << u;
    }
    // With the fields in registers the descriptors go to shared memory (each
    // thread reads its own words back, without conflicts).
    float* const desc = sm + m.desc + 4 * tid;
    float* const desc1 = sm + m.desc + 4 * kResQuads * NT + tid;
    if constexpr (KEEP) {
#pragma unroll
        for (int u = 0; u < kResQuads; ++u) {
            put4(desc + 4 * u * NT, hq_d[u]);
            desc1[u * NT] = __uint_as_float(hq[u]);
        }
#pragma unroll
        for (int u = 0; u < kResScalars; ++u) {
            desc1[(kResQuads + u) * NT] = __uint_as_float(hz[u]);
            desc1[(kResQuads + kResScalars + u) * NT] = hz_d[u];
        }
    }
    auto quad_at = [&](int u) { return KEEP ? __float_as_uint(desc1[u * NT]) : hq[u]; };
    auto scalar_at = [&](int u) { return KEEP ? __float_as_uint(desc1[(kResQuads + u) * NT]) : hz[u]; };
    auto scalar_damp = [&](int u) { return KEEP ? desc1[(kResQuads + kResScalars + u) * NT] : hz_d[u]; };

    // velocities of the own faces of plane l (T: with the tests of faces and
    // gradient orders); x0 .. x3 = P of planes l-1 .. l+2
    auto own_vel = [&](int l, auto tests, const float (&x0)[4], const float (&x1)[4], const float (&x2)[4],
                       const float (&x3)[4], const float (&myz)[5], const float (&myr)[4]) {
        constexpr bool T = decltype(tests)::value;
        const float* const pl = sm + pc + l * PP;
        [[maybe_unused]] const float axl = KEEP ? 0.0f : axs[l0 + l], axr = KEEP ? 0.0f : axs[l0 + l + 1];
        const int gi = i0 + l0 + l;
        const bool x4 = !T || (gi > 0 && gi < g.nx - 2), xex = !T || gi <= g.nx - 2;
        float pm[4], p1[4], p2[4], v[4];
        get4(pl - SP, pm);
        get4(pl + SP, p1);
        get4(pl + 2 * SP, p2);
        const float zl = pl[-1];
        const float2 zr = *reinterpret_cast<const float2*>(pl + 4);
        const float e[7] = {zl, x1[0], x1[1], x1[2], x1[3], zr.x, zr.y};
        if constexpr (!KEEP) get4(sm + xc + l * PX, v);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const float gr = res_grad(cf, x0[t], x1[t], x2[t], x3[t], x4);
            if constexpr (KEEP) v[t] = res_vel(cf, VX[t], gr, DX[t]);
            else v[t] = res_vel(cf, v[t], gr, face_damp(fmaxf(axl, myz[t]), fmaxf(axr, myz[t]), cf.dt));
            if (T && !xex) v[t] = 0.0f;
            if constexpr (KEEP) VX[t] = v[t];
        }
        put4(sm + xc + l * PX, v);
        if constexpr (!KEEP) get4(sm + yc + l * PY, v);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const float gr = res_grad(cf, pm[t], x1[t], p1[t], p2[t], !T || y4);
            if constexpr (KEEP) v[t] = res_vel(cf, VY[t], gr, DY[t]);
            else v[t] = res_vel(cf, v[t], gr, face_damp(fmaxf(axl, myz[t]), fmaxf(axl, myr[t]), cf.dt));
            if (T && !yex) v[t] = 0.0f;
            if constexpr (KEEP) VY[t] = v[t];
        }
        put4(sm + yc + l * PY, v);
        if constexpr (!KEEP) get4(sm + zc + l * PZ, v);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const float gr = res_grad(cf, e[t], e[t + 1], e[t + 2], e[t + 3], !T || (z4 >> t & 1));
            if constexpr (KEEP) v[t] = res_vel(cf, VZ[t], gr, DZ[t]);
            else v[t] = res_vel(cf, v[t], gr, face_damp(fmaxf(axl, myz[t]), fmaxf(axl, myz[t + 1]), cf.dt));
            if (T && !(zex >> t & 1)) v[t] = 0.0f;
            if constexpr (KEEP) VZ[t] = v[t];
        }
        put4(sm + zc + l * PZ, v);
    };
    auto own_vels = [&](auto tests) {
        float myz[5], myr[4], x0[4], x1[4], x2[4], x3[4];
        get4(sm + pc - PP, x0);
        if constexpr (KEEP) {
            get4(sm + pc + PP, x2);
            get4(sm + pc + 2 * PP, x3);
#pragma unroll
            for (int t = 0; t < 4; ++t) x1[t] = P[t];
            own_vel(0, tests, x0, x1, x2, x3, myz, myr);
        } else {
            // max(alpha_y, alpha_z) of the cells, and with the next row's alpha_y
            const float ay = ays[lj], ayr = ays[lj + 1];
            float az[4];
            get4(azs + 4 * qq, az);
#pragma unroll
            for (int t = 0; t < 4; ++t) { myz[t] = fmaxf(ay, az[t]); myr[t] = fmaxf(ayr, az[t]); }
            myz[4] = fmaxf(ay, azs[4 * qq + 4]);
            get4(sm + pc, x1);
            get4(sm + pc + PP, x2);
#pragma unroll 1
            for (int l = 0; l < nl; ++l) {
                get4(sm + pc + (l + 2) * PP, x3);
                own_vel(l, tests, x0, x1, x2, x3, myz, myr);
#pragma unroll
                for (int t = 0; t < 4; ++t) { x0[t] = x1[t]; x1[t] = x2[t]; x2[t] = x3[t]; }
            }
        }
    };
    // P of the own cells of plane l, published (post) when another step follows;
    // x0 .. x3 = Vx of faces l-2 .. l+1, mpz = min of the y and z dampings
    auto own_p = [&](int l, auto tests, const float (&x0)[4], const float (&x1)[4], const float (&x2)[4],
                     const float (&x3)[4], const float (&mpz)[4], uint4* box, unsigned tag, bool post, float amp) {
        constexpr bool T = decltype(tests)::value;
        const float* const yl = sm + yc + l * PY;
        const float* const zl = sm + zc + l * PZ;
        const float px = KEEP ? 1.0f : pxs[l0 + l];
        float ymm[4], ym[4], yp[4], ypp[4], zp[4], p[4], n[4];
        get4(yl - 2 * SV, ymm);
        get4(yl - SV, ym);
        get4(yl + SV, ypp);
        const float2 zb = *reinterpret_cast<const float2*>(zl - 2);
        const float za = zl[4];
        if constexpr (KEEP) {
#pragma unroll
            for (int t = 0; t < 4; ++t) { yp[t] = VY[t]; zp[t] = VZ[t]; p[t] = P[t]; }
        } else {
            get4(yl, yp);
            get4(zl, zp);
            get4(sm + pc + l * PP, p);
        }
        const float e[7] = {zb.x, zb.y, zp[0], zp[1], zp[2], zp[3], za};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const float d1 = fadd(fadd(fsub(x2[t], x1[t]), fsub(yp[t], ym[t])), fsub(e[t + 2], e[t + 1]));
            const float d2 = fadd(fadd(fsub(x3[t], x0[t]), fsub(ypp[t], ymm[t])), fsub(e[t + 3], e[t]));
            const float dv = fadd(fmul(cf.c1, d1), fmul(cf.c2, d2));
            const float pd = KEEP ? PD[KEEP ? t : 0] : fminf(px, mpz[t]);
            n[t] = fmul(fsub(p[t], fmul(cf.bulk, dv)), pd);
            if (T && !(cex >> t & 1)) n[t] = 0.0f;
        }
        if (l == src_l) {   // the pressure the receivers hear, then the next step's sample
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (t == src_t) {
                    s_pre = n[t];
                    if (amp != 0.0f) n[t] = fadd(n[t], amp);
                }
        }
        if constexpr (KEEP) {
#pragma unroll
            for (int t = 0; t < 4; ++t) P[t] = n[t];
        }
        put4(sm + pc + l * PP, n);
        if (post) {
            uint4* const dx = box + 2 * (rx0 + l * BJ * Q);
            uint4* const dy = box + 2 * (ry0 + l * 3 * Q);
            uint4* const dz = box + 2 * (rz0 + l * BJ);
            post4(l0 + l < pxl, dx, n, tag);
            post4(l0 + l >= pxh, dx + 2 * (FX + (3 - bi) * BJ * Q), n, tag);
            post4(pub & 1u, dy, n, tag);
            post4(pub & 2u, dy + 2 * FY, n, tag);
            post4(pub & 4u, dz, n, tag);
            post4(pub & 8u, dz + 2 * FZ, n, tag);
        }
    };
    auto own_ps = [&](auto tests, uint4* box, unsigned tag, bool post, float amp) {
        float mpz[4], x0[4], x1[4], x2[4], x3[4];
        get4(sm + xc - 2 * PX, x0);
        get4(sm + xc - PX, x1);
        if constexpr (KEEP) {
            get4(sm + xc + PX, x3);
#pragma unroll
            for (int t = 0; t < 4; ++t) x2[t] = VX[t];
            own_p(0, tests, x0, x1, x2, x3, mpz, box, tag, post, amp);
        } else {
            const float py = pys[lj];
            get4(pzs + 4 * qq, mpz);
#pragma unroll
            for (int t = 0; t < 4; ++t) mpz[t] = fminf(py, mpz[t]);
            get4(sm + xc, x2);
#pragma unroll 1
            for (int l = 0; l < nl; ++l) {
                get4(sm + xc + (l + 1) * PX, x3);
                own_p(l, tests, x0, x1, x2, x3, mpz, box, tag, post, amp);
#pragma unroll
                for (int t = 0; t < 4; ++t) { x0[t] = x1[t]; x1[t] = x2[t]; x2[t] = x3[t]; }
            }
        }
    };

    uint4* const mine = a.xbuf + 2ll * rec * b;
    const long long parity = 2ll * rec * nbricks;
    const int quad_rounds = min(kResQuads, (FX + FY + NT - 1) / NT), scalar_rounds = min(kResScalars, (3 * FZ + NT - 1) / NT);
    bool ok = true;
    for (int s = 0; s < a.steps; ++s) {
        const bool more = s + 1 < a.steps;
        // the next step's source sample, fetched a phase ahead of its use
        float amp = 0.0f;
        if (src_here && more && s + 1 >= a.dep_from && s + 1 < a.dep_to) amp = __ldg(a.sig + a.step0 + s + 1);
        // ---- the receivers' taps of the step before
        if (s > 0 && s <= a.rec_steps)
            for (int e = tid; e < s_ntap; e += NT)
                a.tap_out[(long long)(s - 1) * a.n_taps + taps[e].y] = taps[e].x >= 0 ? sm[taps[e].x] : s_pre;

        // ---- velocities of the own faces
        if (nl > 0) {
            if (fast) own_vels(std::false_type{});
            else own_vels(std::true_type{});
        }
        // ---- velocities of the halo faces
#pragma unroll
        for (int u = 0; u < kResQuads; ++u)
            if (u < quad_rounds && (hq_on >> u & 1)) {
                const unsigned at = quad_at(u);
                const float* const pl = sm + 4 * (at & 0xFFFFu);
                float* const vl = sm + 4 * (at >> 16);
                float d[4];
                if constexpr (KEEP) get4(desc + 4 * u * NT, d);
                else
#pragma unroll
                    for (int t = 0; t < 4; ++t) d[t] = hq_d[u][t];
                const int st = hq_y >> u & 1 ? SP : PP;
                float pm[4], p0[4], p1[4], p2[4], v[4];
                get4(pl - st, pm);
                get4(pl, p0);
                get4(pl + st, p1);
                get4(pl + 2 * st, p2);
                get4(vl, v);
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    v[t] = res_vel(cf, v[t], res_grad(cf, pm[t], p0[t], p1[t], p2[t], hq_4 >> u & 1), d[t]);
                put4(vl, v);
            }
#pragma unroll
        for (int u = 0; u < kResScalars; ++u)
            if (u < scalar_rounds && (hz_on >> u & 1)) {
                const unsigned at = scalar_at(u);
                const float* const pl = sm + (at & 0xFFFFu);
                float* const vl = sm + (at >> 16);
                *vl = res_vel(cf, *vl, res_grad(cf, pl[-1], pl[0], pl[1], pl[2], hz_4 >> u & 1), scalar_damp(u));
            }
        __syncthreads();

        // ---- P of the own cells, published as it is computed
        const unsigned tag = a.epoch + (unsigned)s + 1u;
        if (nl > 0) {
            uint4* const box = mine + (s & 1 ? parity : 0);
            const bool post = more && b != a.hold_brick;
            if (fast) own_ps(std::false_type{}, box, tag, post, amp);
            else own_ps(std::true_type{}, box, tag, post, amp);
        }
        // ---- the neighbours' layers into the halo: all of a thread's records in
        // flight together, polled until each carries this step's number
        if (more) {
            const uint4* const base = a.xbuf + (s & 1 ? parity : 0);
            unsigned left = r_mask;
            unsigned long long t0 = 0;
            for (int it = 0; left && ok; ++it) {
                Record w[kResRecords];
#pragma unroll
                for (int u = 0; u < kResRecords; ++u) w[u].load(left >> u & 1, base + 2 * (r_at[u] >> 13));
#pragma unroll
                for (int u = 0; u < kResRecords; ++u) {
                    const bool in = (left >> u & 1) && w[u].landed(tag);
                    w[u].store(in, sm + m.p + 4 * (r_at[u] & 0x1FFFu));
                    left &= ~((unsigned)in << u);
                }
                if ((it & 63) == 63) {   // a long wait: its bounds
                    const unsigned long long now = global_ns();
                    if (t0 == 0) t0 = now;
                    if (now - t0 > 1000ull * a.wait_us || it > kWaitPolls ||
                        *reinterpret_cast<const volatile unsigned*>(a.status + kStatusTimeout) != 0xFFFFFFFFu)
                        ok = false;
                }
            }
        }
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicMin(a.status + kStatusTimeout, (unsigned)b);
            return;
        }
    }
    // ---- the last step's taps, and the fields back to memory (zeros beyond Nz)
    if (a.steps <= a.rec_steps)
        for (int e = tid; e < s_ntap; e += NT)
            a.tap_out[(long long)(a.steps - 1) * a.n_taps + taps[e].y] = taps[e].x >= 0 ? sm[taps[e].x] : s_pre;
    for (int l = 0; l < nl; ++l) {
        const int src[4] = {pc + l * PP, xc + l * PX, yc + l * PY, zc + l * PZ};
        float* const dst[4] = {a.pn, a.vout[0], a.vout[1], a.vout[2]};
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            float v[4];
            get4(sm + src[f], v);
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (!(cex >> t & 1)) v[t] = 0.0f;
            put4(dst[f] + gid + l * g.plane, v);
        }
    }
}

// The receivers' rows from their recorded taps, in the samplers' tap order.
__global__ void k_tap_rows(const float* __restrict__ tap, const float* __restrict__ w, int rows, int n_rec,
                           float* __restrict__ out)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= rows * n_rec) return;
    const float* v = tap + 8ll * q;
    const float* ww = w + 8 * (q % n_rec);
    float s = fmul(ww[0], v[0]);
    for (int t = 1; t < 8; ++t) s = fadd(s, fmul(ww[t], v[t]));
    out[q] = s;
}

template <class B>
ResMap map_of(int L, int bi, int n_taps)
{
    ResMap m;
    int o = 0;
    auto add = [&](int n) { const int at = o; o += (n + 3) / 4 * 4; return at; };
    m.p = add((bi + 6) * B::PP);
    m.vx = add((bi + 3) * B::PX);
    m.vy = add(bi * B::PY);
    m.vz = add(bi * B::PZ);
    m.ax = add(bi + 4);
    m.ay = add(B::BJ + 4);
    m.az = add(B::BK + 8);
    m.px = add(bi);
    m.py = add(B::BJ);
    m.pz = add(B::BK);
    m.taps = add(2 * n_taps);
    m.desc = add(L == 1 ? kResThreads * (5 * kResQuads + 2 * kResScalars) : 0);
    m.total = o;
    return m;
}

template <bool KEEP, class B>
cudaError_t launch_of(ResArgs& a, int n_taps, bool refuse, cudaStream_t s)
{
    static std::atomic<unsigned long long> ready{0};   // devices whose shared-memory limit is raised
    const void* const fn = (const void*)k_resident<KEEP, B>;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !(ready.load() >> dev & 1)) {
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem);
        if (e != cudaSuccess) return e;
        if (dev < 64) ready |= 1ull << dev;
    }
    a.m = map_of<B>(a.L, a.bi, n_taps);
    void* args[] = {&a};
    const dim3 grid(refuse ? 1u << 24 : a.nbi * a.nbj * a.nbk), block(kResThreads);
    return cudaLaunchCooperativeKernel(fn, grid, block, args, 4 * (size_t)a.m.total, s);
}

// The compiled bricks (quads x rows), narrow ones for small rooms.
template <class F>
bool for_brick(int q, int bj, F f)
{
    if (q == 2 && bj == 8) return f(Brick<2, 8>{});
    if (q == 4 && bj == 8) return f(Brick<4, 8>{});
    if (q == 4 && bj == 16) return f(Brick<4, 16>{});
    if (q == 8 && bj == 8) return f(Brick<8, 8>{});
    if (q == 8 && bj == 16) return f(Brick<8, 16>{});
    return false;
}
// Estimated time of a step in quads: measured steps of 40 cuts of rooms from
// 32^3 to 128x96x96 lie within 6 % of 1.5 us (the exchange and the barriers)
// plus 2.3 ns per own and halo quad of a brick (64^3: 3.55 us, 96^3: 6.5,
// 128x96x96: 7.9); fewer planes per thread win ties.
double resident_cost(int L, int bi, int bj, int q)
{
    const double own = (double)bi * bj * q, halo = 3.0 * (bj * q + bi * q + bi * bj / 4.0);
    return own + halo + 20.0 * L;
}

constexpr int kBricks[][2] = {{2, 8}, {4, 8}, {4, 16}, {8, 8}, {8, 16}};

}  // namespace

// The bricks of a room: the cut of the least estimated step time among those
// with at most one brick per SM whose threads, halo items, exchange records and
// shared memory stay inside the kernel's limits.  Bricks that a neighbour reads
// from must be three planes deep.
ResPlan resident_plan(const Grid& g, int sms)
{
    ResPlan best;
    if (g.nx < 1 || g.ny < 1 || g.nz < 1) return best;
    double least = 1e30;
    for (const auto& q_bj : kBricks) {
        const int q = q_bj[0], bj = q_bj[1];
        const int nbk = (g.nz + 4 * q - 1) / (4 * q), nbj = (g.ny + bj - 1) / bj;
        if ((long long)nbk * nbj > sms) continue;
        for (int nbi = 1; nbi <= std::min(g.nx, sms / (nbk * nbj)); ++nbi) {
            const int bi = (g.nx + nbi - 1) / nbi;
            if ((g.nx + bi - 1) / bi != nbi || (nbi > 1 && bi < 3)) continue;
            const int runs = kResThreads / (bj * q), L = (bi + runs - 1) / runs;
            const int fx = 3 * bj * q, fy = 3 * bi * q, fz = bi * bj, rec = 2 * (fx + fy + fz);
            if (fx + fy > kResQuads * kResThreads || 3 * fz > kResScalars * kResThreads ||
                rec > kResRecords * kResThreads || (long long)rec * nbi * nbj * nbk >= 1 << 19)
                continue;
            int total = 0, p_quads = 0;
            for_brick(q, bj, [&](auto B) {
                using T = decltype(B);
                total = map_of<T>(L, bi, kResMaxTaps).total;
                p_quads = (bi + 6) * T::PP / 4;
                return true;
            });
            if (4 * total > kResSmem || p_quads > 1 << 13) continue;
            const double cost = resident_cost(L, bi, bj, q);
            if (cost < least) {
                least = cost;
                best.ok = true;
                best.L = L; best.bi = bi; best.bj = bj; best.q = q;
                best.nbi = nbi; best.nbj = nbj; best.nbk = nbk;
                best.xbytes = 64ull * rec * nbi * nbj * nbk;
            }
        }
    }
    return best;
}

int resident_max_taps() { return kResMaxTaps; }

cudaError_t launch_resident(const FusedArgs& f, const ResPlan& pl, int steps, void* xbuf, unsigned epoch, int dep_from,
                            int dep_to, const long long* tap_idx, int n_taps, int rec_steps, float* tap_out,
                            cudaStream_t s)
{
    ResArgs a{};
    a.g = f.g; a.cf = f.cf; a.tb = f.tb;
    a.p = f.p; a.pn = f.pn;
    for (int c = 0; c < 3; ++c) { a.vin[c] = f.vin[c]; a.vout[c] = f.vout[c]; }
    a.status = f.status;
    a.wait_us = f.wait_us;
    a.hold_brick = f.hold_brick;
    a.L = pl.L; a.bi = pl.bi;
    a.nbi = pl.nbi; a.nbj = pl.nbj; a.nbk = pl.nbk;
    a.xbuf = static_cast<uint4*>(xbuf);
    a.epoch = epoch;
    a.steps = steps;
    a.sig = f.dep_sig;
    a.step0 = f.dep_step;
    a.dep_from = dep_from; a.dep_to = dep_to;
    a.si = f.dep_i; a.sj = f.dep_j; a.sk = f.dep_k;
    a.tap_idx = tap_idx; a.n_taps = n_taps; a.rec_steps = rec_steps; a.tap_out = tap_out;
    cudaError_t e = cudaErrorInvalidValue;
    for_brick(pl.q, pl.bj, [&](auto B) {
        using T = decltype(B);
        e = pl.L == 1 ? launch_of<true, T>(a, n_taps, f.refuse, s) : launch_of<false, T>(a, n_taps, f.refuse, s);
        return true;
    });
    return e;
}

cudaError_t launch_tap_rows(const float* tap, const float* w, int rows, int n_rec, float* out, cudaStream_t s)
{
    const int n = rows * n_rec;
    if (n <= 0) return cudaSuccess;
    k_tap_rows<<<(n + 127) / 128, 128, 0, s>>>(tap, w, rows, n_rec, out);
    return cudaGetLastError();
}

}  // namespace fdtd
