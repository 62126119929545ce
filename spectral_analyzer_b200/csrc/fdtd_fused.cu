/*
 * fdtd_fused.cu — single-pass velocity+pressure step for open rooms (and, with
 * the walled rules of the two-pass kernels, for large walled scenes).
 *
 * One launch advances V^{n-1/2} -> V^{n+1/2} and P^n -> P^{n+1} over the whole
 * grid, reading each field once and writing each once: 16 B read + 16 B
 * written per cell-update, the HBM floor of the scheme (the two-pass step
 * moves 48 B).
 *
 * Decomposition (2.5D): a CTA owns a TJ x 128 tile of (j, k) columns — one warp
 * per row j, four consecutive k per lane (float4) — and marches along i over a
 * segment [i_beg, i_end).  Iteration u of the march
 *   - computes the new Vx on face f = u-2 of the own columns from P^n planes
 *     f-1 .. f+2 and keeps the last four faces in a register queue;
 *   - computes, for plane i = u-3, the new Vy of rows j0-2 .. j0+TJ and the new
 *     Vz of faces k0-2 .. k0+128: faces outside the tile are recomputed here
 *     from V^{n-1/2}, never read back from a neighbour, so the step writes the
 *     other velocity set;
 *   - finishes P^{n+1} of plane i from the 4th-order divergence.
 *
 * Loads: one thread per CTA issues four TMA boxes per plane (P with a 3-cell
 * halo in j and a 4-cell halo in k, Vx, Vy with its halo rows, Vz with its halo
 * columns) into a ring of shared-memory stages D planes ahead of use, each
 * stage completed by an mbarrier; boxes that reach outside the grid are
 * zero-filled by the TMA unit.  The box origin in k is k0-4 or k0, a multiple
 * of 4 floats (16 bytes).  Every mbarrier wait is bounded: a wait that runs
 * out sets a status word, the CTA drains its copies in flight (again bounded)
 * and returns.  Halo rows and columns are shared with neighbouring CTAs that
 * march at the same pace, so they are served mostly from L2.
 *
 * Absorption: on x-interior planes (alpha_x = 0, all but the 2*n_pml PML
 * planes) a face's damping depends on (j, k) only and is a per-thread constant
 * computed once; PML planes take a general path that computes it per face.
 * Both evaluate the same expression, so results do not depend on the path.
 *
 * Arithmetic is the reference's (csrc/kernels/acoustic_fdtd.cpp:1099-1148 for
 * the velocity, :894-952 and :1176-1234 for the pressure) with every operation
 * separately rounded (fadd/fsub/fmul): bit-identical to the two-pass kernels
 * and to the reference.
 */
#include "fdtd_internal.h"
#include "fdtd_tma.h"
#include "launch.h"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>
#include <type_traits>
#include <vector>

namespace fdtd {

namespace {

// TJ rows x TK = 4*LW columns per CTA; LW threads per row (float4 each), so a
// warp covers 32/LW rows.
template <int TJ_, int D_, int LW_ = 32>
struct Cfg {
    static constexpr int TJ = TJ_;              // rows per CTA
    static constexpr int LW = LW_;              // threads per row
    static constexpr int RW = 32 / LW;          // rows per warp
    static constexpr int TK = 4 * LW;           // columns per CTA
    static constexpr int D = D_;                // prefetch distance (iterations)
    static constexpr int NT = 32 * (TJ / RW);
    static constexpr int HW = (3 * TJ + 31) / 32;   // warps computing the halo Vz faces
    static constexpr int PR = TJ + 6;           // P box rows j0-3 .. j0+TJ+2
    static constexpr int PC = TK + 8;           // P box cols k0-4 .. k0+TK+3
    static constexpr int RING = D + 4;          // planes u-3 .. u in use + D in flight
    static constexpr int VYR = TJ + 3;          // Vy rows j0-2 .. j0+TJ
    // box sizes in floats, and stage strides rounded to 128 bytes
    static constexpr int P_BOX = PR * PC;
    static constexpr int VX_BOX = TJ * TK;
    static constexpr int VY_BOX = VYR * TK;
    static constexpr int VZ_BOX = TJ * PC;      // Vz cols k0-4 .. k0+TK+3
    static constexpr int r32(int n) { return (n + 31) / 32 * 32; }
    static constexpr int P_STAGE = r32(P_BOX);
    static constexpr int VX_OFF = 0;
    static constexpr int VY_OFF = r32(VX_BOX);
    static constexpr int VZ_OFF = VY_OFF + r32(VY_BOX);
    static constexpr int V_STAGE = VZ_OFF + r32(VZ_BOX);
    static constexpr int VSTAGES = D + 1;
    static constexpr int AY_N = TJ + 4;         // alpha_y rows j0-2 .. j0+TJ+1
    // shared-memory map (floats from a 128-byte aligned base)
    static constexpr int RING0 = 0;
    static constexpr int VST0 = RING0 + RING * P_STAGE;
    static constexpr int VYN0 = VST0 + VSTAGES * V_STAGE;
    static constexpr int VZN0 = VYN0 + r32(VY_BOX);
    static constexpr int AY0 = VZN0 + r32(VZ_BOX);
    static constexpr int AZ0 = AY0 + r32(AY_N);
    static constexpr int BAR0 = AZ0 + r32(PC);  // RING mbarriers (8 B each)
    static constexpr int SMEM_FLOATS = BAR0 + 2 * RING;
    static constexpr size_t SMEM_BYTES = sizeof(float) * SMEM_FLOATS + 128;   // + base alignment
    static constexpr unsigned P_BYTES = 4u * P_BOX;
    static constexpr unsigned VX_BYTES = 4u * VX_BOX;
    static constexpr unsigned VYZ_BYTES = 4u * (VY_BOX + VZ_BOX);
    static_assert((PC * 4) % 16 == 0 && (TK * 4) % 16 == 0, "TMA box rows are 16-byte multiples");
    static_assert(PC <= 256 && PR <= 256 && VYR <= 256, "TMA box extent");
    static_assert(VYR <= 2 * TJ, "at most two Vy rows per warp");
    static_assert(LW == 32 || LW == 16, "a row is one warp or half a warp");
    static_assert(TJ % RW == 0 && HW * 32 <= NT, "whole warps of rows; halo warps exist");
};

__device__ __forceinline__ float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void sts4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void stg4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float& at(float4& v, int q) { return reinterpret_cast<float*>(&v)[q]; }
__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
// a face whose open fraction is 0 is closed
__device__ __forceinline__ float4 close4(float4 v, const float4& fr)
{
    if (fr.x == 0.0f) v.x = 0.0f;
    if (fr.y == 0.0f) v.y = 0.0f;
    if (fr.z == 0.0f) v.z = 0.0f;
    if (fr.w == 0.0f) v.w = 0.0f;
    return v;
}
__device__ __forceinline__ float4 mul4(const float4& v, const float4& fr)
{
    return make_float4(fmul(v.x, fr.x), fmul(v.y, fr.y), fmul(v.z, fr.z), fmul(v.w, fr.w));
}

// staggered gradient: 4th order in the interior of the face range, else 2nd
__device__ __forceinline__ float grad4(const Coef& cf, float pm, float p0, float p1, float p2, bool fourth)
{
    // both orders, then a selection: a branch per face costs more than the products
    const float d = fsub(p1, p0), w = fadd(fmul(cf.c1, d), fmul(cf.c2, fsub(p2, pm)));
    return fourth ? w : d;
}

// V^{n+1/2} = (V^{n-1/2} - vc*grad) * damp
__device__ __forceinline__ float vupd(const Coef& cf, float vold, float grad, float damp)
{
    return fmul(fsub(vold, fmul(cf.vc, grad)), damp);
}

// four faces, 4th-order gradient, given damping (the x-interior fast path)
__device__ __forceinline__ float4 vel4(const Coef& cf, const float4& pm, const float4& p0,
                                      const float4& p1, const float4& p2, const float4& vo,
                                      const float4& dmp)
{
    float4 r;
    r.x = vupd(cf, vo.x, grad4(cf, pm.x, p0.x, p1.x, p2.x, true), dmp.x);
    r.y = vupd(cf, vo.y, grad4(cf, pm.y, p0.y, p1.y, p2.y, true), dmp.y);
    r.z = vupd(cf, vo.z, grad4(cf, pm.z, p0.z, p1.z, p2.z, true), dmp.z);
    r.w = vupd(cf, vo.w, grad4(cf, pm.w, p0.w, p1.w, p2.w, true), dmp.w);
    return r;
}

// as vel4, with a per-face gradient order (bit q of m4) and existence (bit q of ok)
__device__ __forceinline__ float4 vel4_masked(const Coef& cf, float4 pm, float4 p0, float4 p1,
                                             float4 p2, float4 vo, float4 dmp, int m4, int ok)
{
    float4 r;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float gr = grad4(cf, at(pm, q), at(p0, q), at(p1, q), at(p2, q), (m4 >> q) & 1);
        const float v = vupd(cf, at(vo, q), gr, at(dmp, q));
        at(r, q) = ((ok >> q) & 1) ? v : 0.0f;
    }
    return r;
}

// General-path velocity of four faces: damping from the alphas (PML planes
// and ragged tiles).  Inlined: an out-of-line call here cost the fast path
// about 9 % more instructions through the call's register traffic.
__device__ __forceinline__ float4 vel4_general(Coef cf, float4 pm, float4 p0, float4 p1, float4 p2,
                                            float4 vo, float4 aL, float4 aR, int m4, int ok)
{
    float4 dmp;
#pragma unroll
    for (int q = 0; q < 4; ++q) at(dmp, q) = face_damp(at(aL, q), at(aR, q), cf.dt);
    return vel4_masked(cf, pm, p0, p1, p2, vo, dmp, m4, ok);
}

// P^{n+1} = (P^n - bulk*div) * pd, div = c1*(dx+dy+dz) + c2*(dxx+dyy+dzz)
__device__ __forceinline__ float pupd(const Coef& cf, float p, float xp, float xm, float xpp,
                                      float xmm, float yp, float ym, float ypp, float ymm, float zp,
                                      float zm, float zpp, float zmm, float pd)
{
    const float d1 = fadd(fadd(fsub(xp, xm), fsub(yp, ym)), fsub(zp, zm));
    const float d2 = fadd(fadd(fsub(xpp, xmm), fsub(ypp, ymm)), fsub(zpp, zmm));
    const float dv = fadd(fmul(cf.c1, d1), fmul(cf.c2, d2));
    return fmul(fsub(p, fmul(cf.bulk, dv)), pd);
}

// Load-pipeline state carried by a CTA from one tile to the next: the ring slot
// of the next plane and V stage to be loaded, and the mbarrier parity to wait
// for next, per ring slot.  Between tiles every issued load has been consumed.
struct Pipe {
    int ps = 0, vs = 0;
    unsigned ph = 0;
};

template <class C>
__device__ __forceinline__ unsigned smem_base_u32(float** smem_out)
{
    // an offset from the array, not a pointer made from an integer: the compiler
    // must see shared memory, or every access becomes a generic one with 64-bit
    // addresses (512x384x256 room: 313 us per step)
    extern __shared__ __align__(128) float smem_raw[];
    float* const smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u) / 4u;
    *smem_out = smem;
    return smem_u32(smem);
}

template <class C>
__device__ __forceinline__ void init_barriers(unsigned bar0)
{
    if (threadIdx.x == 0) {
        for (int q = 0; q < C::RING; ++q) mbar_init(bar0 + 8u * q, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
}

// One tile (TJ x TK columns, own planes [first, first + len)) of the fused step.
// Returns false when a load wait ran out (the CTA must stop; status is set).
// PEER = false compiles out the neighbour ghost-plane stores (single rooms and
// batches), which the slab step of a split room needs.  WALLS = true adds the
// walled-scene rules of the two-pass kernels to the general body: a face whose
// open fraction is 0 is closed (its new velocity is 0), the divergence sees
// each face's velocity times its fraction (when fractions were set), and
// solid cells keep P = 0, in both the interior and the general body.  start()
// runs before the first load (it waits for what the loads read) and says what
// to do once the first loads are on their way.
template <class C, bool PEER = true, bool WALLS = false, class Start>
__device__ __forceinline__ bool fused_tile(const FusedArgs& a, const CUtensorMap* tmP,
                                           const CUtensorMap* tmX, const CUtensorMap* tmY,
                                           const CUtensorMap* tmZ, int tile, int first, int len,
                                           int tiles_k, float* smem, unsigned sbase, unsigned bar0,
                                           Pipe& pp, Start start)
{
    float* const vyn = smem + C::VYN0;
    float* const vzn = smem + C::VZN0;
    float* const ay_s = smem + C::AY0;
    float* const az_s = smem + C::AZ0;

    const Grid g = a.g;
    const int nx = g.nx, ny = g.ny, nz = g.nz, sz = g.sz;
    const long long PL = g.plane;
    // lane = this thread's float4 column in its row, w = its row in the tile
    // (with 32 threads per row: the hardware lane and warp)
    const int tid = threadIdx.x, lane = tid % C::LW, w = tid / C::LW;
    const int tk = tile % tiles_k, tj = tile / tiles_k;
    const int j0 = tj * C::TJ, k0 = tk * C::TK;
    // own planes and the global frame (a slab of a split room, or the whole room)
    const bool slab = a.xs.nxg > 0;
    const int nxg = slab ? a.xs.nxg : nx, xg0 = slab ? a.xs.xg0 : 0;
    const int own_lo = slab ? a.xs.i_lo : 0, own_hi = slab ? a.xs.i_lo + a.xs.n_own : nx;
    const int i_beg = own_lo + first;
    if (i_beg >= own_hi) return true;
    const int i_end = min(i_beg + len, own_hi);
    const Coef cf = a.cf;

    __syncthreads();   // the previous tile's readers of the tables are done
    for (int e = tid; e < C::AY_N; e += C::NT) {
        const int j = j0 - 2 + e;
        ay_s[e] = (j >= 0 && j < ny) ? __ldg(a.tb.ay + j) : 0.0f;
    }
    for (int e = tid; e < C::PC; e += C::NT) {
        const int k = k0 - 4 + e;
        az_s[e] = (k >= 0 && k < nz) ? __ldg(a.tb.az + k) : 0.0f;
    }
    __syncthreads();

    // Loads feeding iteration u (issued by one thread): P plane u, Vx face u-2,
    // Vy/Vz of plane u-3, all on the plane's mbarrier.
    auto issue = [&](int u, int ps, int vsg) {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        const unsigned pb = bar0 + 8u * ps;
        const int f = u - 2, io = u - 3, fg = f + xg0;
        const bool vx = (u >= i_beg && fg >= 0 && fg <= nxg - 2);
        const bool vyz = (io >= i_beg && io < i_end);
        mbar_expect_tx(pb, C::P_BYTES + (vx ? C::VX_BYTES : 0u) + (vyz ? C::VYZ_BYTES : 0u));
        if (u != a.hold_plane)
            tma_load3(sbase + 4u * (C::RING0 + ps * C::P_STAGE), tmP, k0 - 4, j0 - 3, u, pb);
        const unsigned vdst = sbase + 4u * (C::VST0 + vsg * C::V_STAGE);
        if (vx) tma_load3(vdst + 4u * C::VX_OFF, tmX, k0, j0, f, pb);
        if (vyz) {
            tma_load3(vdst + 4u * C::VY_OFF, tmY, k0, j0 - 2, io, pb);
            tma_load3(vdst + 4u * C::VZ_OFF, tmZ, k0 - 4, j0, io, pb);
        }
    };

    auto started = start();
    const int u0 = i_beg - 3, u1 = i_end + 2;
    // Plane v of the march lives in ring slot (ps + v - u0) mod RING, iteration
    // v's V data in stage (vs + v - u0) mod VSTAGES: at iteration u planes u-3
    // .. u are in use, u+1 .. u+D-1 in flight, and the slots of u+D (held by
    // plane u-4 and iteration u-1 before) are free.
    int ps = pp.ps, vs0 = pp.vs;
    unsigned ph = pp.ph;
    auto ring = [&](int q) { return q >= C::RING ? q - C::RING : q; };
    auto vring = [&](int q) { return q >= C::VSTAGES ? q - C::VSTAGES : q; };
    // the issuing thread is in a warp without a second Vy row or halo Vz faces
    const bool issuer = tid == C::NT / 2;
    if (issuer)
        for (int q = 0; q < C::D; ++q) issue(u0 + q, ring(ps + q), vring(vs0 + q));
    started();
    // stage offsets (floats) of planes u-3 .. u, rotated each iteration
    int o0 = ps * C::P_STAGE, o1 = 0, o2 = 0, o3 = 0;
    {
        int q = ps;
        q = q == 0 ? C::RING - 1 : q - 1; o1 = q * C::P_STAGE;
        q = q == 0 ? C::RING - 1 : q - 1; o2 = q * C::P_STAGE;
        q = q == 0 ? C::RING - 1 : q - 1; o3 = q * C::P_STAGE;
    }

    // ---- per-thread constants of the own row and columns
    const int jr = j0 + w;
    const int kb = k0 + 4 * lane;                 // first own k
    const bool row_ok = jr < ny;
    const bool kfull = k0 + C::TK <= nz;          // every own k of the CTA is a cell
    const bool st_ok = row_ok && kb < sz;         // the float4 store stays inside the row
    const int own = row_ok ? jr * sz + kb : 0;    // in-plane offset of the own float4
    const int cP = (w + 3) * C::PC + 4 * lane + 4;    // own cells in a P stage
    int zm4 = 0, zok = 0;                         // own Vz faces: 4th order / existing
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int kf = kb + q;
        zm4 |= (kf > 0 && kf < nz - 2) ? (1 << q) : 0;
        zok |= (kf <= nz - 2) ? (1 << q) : 0;
    }
    float4 myz, mpz, dxi, dzi;
    {
        const float pyj = row_ok ? __ldg(a.tb.py + jr) : 1.0f;
        const float ayj = ay_s[w + 2];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = kb + q;
            const float azk = az_s[4 * lane + 4 + q];
            at(myz, q) = fmaxf(ayj, azk);
            at(mpz, q) = fminf(pyj, k < nz ? __ldg(a.tb.pz + k) : 1.0f);
            at(dxi, q) = face_damp(at(myz, q), at(myz, q), cf.dt);
            at(dzi, q) = face_damp(fmaxf(ayj, azk), fmaxf(ayj, az_s[4 * lane + 5 + q]), cf.dt);
        }
    }
    // Vy items of this thread: row w (all warps) and row TJ+w (the first VYR-TJ warps)
    constexpr int NY_IT = 2;
    float4 dyi[NY_IT];
#pragma unroll
    for (int m = 0; m < NY_IT; ++m) {
        const int r = m == 0 ? w : C::TJ + w;
        dyi[m] = make_float4(1.f, 1.f, 1.f, 1.f);
        if (r < C::VYR) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float azk = az_s[4 * lane + 4 + q];
                at(dyi[m], q) = face_damp(fmaxf(ay_s[r], azk), fmaxf(ay_s[r + 1], azk), cf.dt);
            }
        }
    }
    float4 qx0 = make_float4(0.f, 0.f, 0.f, 0.f), qx1 = qx0, qx2 = qx0, qx3 = qx0;
    int u_fail = u1 + 1;   // iteration whose wait ran out (none)
    // alpha_x / px window: at iteration u, axw{3,2,1,0} = alpha_x[u-3 .. u] and
    // pxw = px[u-3]; the next iteration's values are prefetched one iteration ahead
    auto ax_at = [&](int q) { return (q >= 0 && q < nx) ? __ldg(a.tb.ax + q) : 0.0f; };
    auto px_at = [&](int q) { return (q >= 0 && q < nx) ? __ldg(a.tb.px + q) : 1.0f; };
    float axw3 = ax_at(u0 - 3), axw2 = ax_at(u0 - 2), axw1 = ax_at(u0 - 1), axw0 = ax_at(u0);
    float pxw = px_at(u0 - 3);

    // The interior iterations take a separately compiled body without the
    // general path (the general path
    // present in the loop costs the interior about 12 % although it never runs
    // there).  Iteration u is interior when plane u-3 and faces u-2 .. u-1 have
    // no x absorption, face u-2 has the 4th-order gradient and the planes u-3,
    // u-2 are own ones.  Rows beyond the room and Vy faces at the j ends are
    // warp-uniform cases the interior body handles itself; columns beyond the
    // room (a partial k tile) hold zero pressure and velocity, so their faces
    // come out zero, their stores end at the row's padding and their cells are
    // set to zero (with the general body on partial tiles the 160x128x112 room,
    // one partial tile wide, took 31.0 us per step).  Both bodies
    // evaluate the same expressions (alpha_x = 0, px = 1 there), so the results
    // do not depend on the choice.  The step runs in one wave, so a CTA left on
    // the general body for its whole march would set the kernel's time.
    int fast_lo = u1 + 1, fast_hi = u1 + 1;
    if (a.tb.xi_hi > a.tb.xi_lo) {
        fast_lo = max(max(a.tb.xi_lo + 3, 3 - xg0), i_beg + 3);
        fast_hi = min(min(a.tb.xi_hi + 1, nxg - xg0), u1 + 1);
        if (fast_lo >= fast_hi) fast_lo = fast_hi = u1 + 1;
    }

    // What the interior body needs of this thread's items, worked out once: the
    // existence and gradient order of its Vy faces (jmid: every Vy face of the
    // tile exists and is of 4th order), its halo Vz face (offsets of P in a P
    // stage and of the velocity in a V stage, order, damping), the iteration
    // whose plane receives the source sample in this CTA, and the places of its
    // results in memory, advanced plane by plane.
    const bool jmid = j0 - 2 > 0 && j0 + C::TJ < ny - 2;
    const int jfa = j0 - 2 + w, jfb = j0 - 2 + C::TJ + w;
    const bool ya_ok = jfa >= 0 && jfa <= ny - 2, yb_ok = jfb >= 0 && jfb <= ny - 2;
    const bool ya_4 = jfa > 0 && jfa < ny - 2, yb_4 = jfb > 0 && jfb < ny - 2;
    const int hl = tid - (C::NT - 32 * C::HW);
    const int h_j = hl / 3, h_c = hl - 3 * h_j < 2 ? 2 + hl - 3 * h_j : C::TK + 4, h_k = k0 - 4 + h_c;
    const bool h_mine = hl >= 0 && hl < 3 * C::TJ, h_ok = h_mine && j0 + h_j < ny && h_k >= 0 && h_k <= nz - 2;
    const bool h_4 = h_k > 0 && h_k < nz - 2;
    float h_d = 1.0f;
    if (h_ok) h_d = face_damp(fmaxf(ay_s[h_j + 2], az_s[h_c]), fmaxf(ay_s[h_j + 2], az_s[h_c + 1]), cf.dt);
    const int h_p = (h_j + 3) * C::PC + h_c, h_v = h_j * C::PC + h_c;
    int dep_u = kNoPlane, dep_at = 0;
    if (a.dep_sig && tid == 0) {
        const int dj = a.dep_j - (j0 - 3), dk = a.dep_k - (k0 - 4);
        if (dj >= 0 && dj < C::PR && dk >= 0 && dk < C::PC) {
            dep_u = a.dep_i;
            dep_at = dj * C::PC + dk;
        }
    }
    float *gX = nullptr, *gYa = nullptr, *gYb = nullptr, *gZ = nullptr, *gP = nullptr;
    // WALLS: the wall codes of the groups whose fractions iteration u reads (Vx
    // face u-2 and plane u-3), the plate node (at plane 0) whose faces lie in this
    // thread's quad (-1: none), and whether its halo face is a plate's
    unsigned wc_x = 0u, wc_a = 0u, wc_b = 0u, wc_z = 0u;
    const uint8_t* wr = nullptr;      // a.walls at plane u-2, advanced with u
    const int pl4 = (int)(PL >> 2), own4 = own >> 2, ya4 = ((jfa * sz + kb) >> 2) - pl4, yb4 = ((jfb * sz + kb) >> 2) - pl4;
    const bool wx_on = st_ok, wa_on = ya_ok && kb < sz, wb_on = yb_ok && kb < sz && C::TJ + w < C::VYR;
    auto wall_codes = [&](int u) {    // wr at plane u-2
        const bool in = u - 3 >= i_beg && u - 3 < i_end;
        wc_x = wx_on && (unsigned)(u - 2) < (unsigned)nx ? __ldg(wr + own4) : 0u;
        wc_a = wa_on && in ? __ldg(wr + ya4) : 0u;
        wc_b = wb_on && in ? __ldg(wr + yb4) : 0u;
        wr += pl4;
    };
    int pl_node = -1;
    bool pl_halo = false;
    if constexpr (WALLS) {
        const int iz = a.plate.iz;
        if (a.plate.code && row_ok && kb <= iz && iz - 1 <= kb + 3) pl_node = jr;
        pl_halo = a.plate.code && h_ok && (h_k == iz - 1 || h_k == iz);
        wr = a.walls + (long long)(u0 - 3) * pl4;
        wall_codes(u0 - 1);
        wc_z = wc_x;
        wall_codes(u0);
    }
    // a plate face takes the plate's velocity after the update
    auto plate_face = [&](float v, int k, unsigned c, float vp) {
        return ((k == a.plate.iz - 1 && (c & 1u)) || (k == a.plate.iz && (c & 2u))) ? vp : v;
    };

    // One iteration of the march; FAST = the interior body.  False when a load
    // wait ran out (u_fail is then set).
    auto iteration = [&](const int u, auto fast_tag) -> bool {
        constexpr bool FAST = decltype(fast_tag)::value;
        // wait for plane u (P) and iteration u's V data; the decision to stop on a
        // timeout is made by the whole CTA (the barrier below is also the one that
        // separates the previous iteration's reads from this iteration's writes)
        // WALLS: this iteration's face fractions and solid flags, where the groups'
        // wall codes (read an iteration ahead) call for them, loaded before the
        // wait so that their latency overlaps it; and the plate's face velocity
        [[maybe_unused]] float4 pf_x = make_float4(1.f, 1.f, 1.f, 1.f), pf_y0 = pf_x, pf_y1 = pf_x, pf_z = pf_x;
        [[maybe_unused]] float pf_h = 1.0f, pl_w = 0.0f, pl_wp = 0.0f, pl_hw = 0.0f, pl_hwp = 0.0f;
        [[maybe_unused]] unsigned pf_s = 0u, pl_c = 0u, pl_hc = 0u;
        [[maybe_unused]] const unsigned cx = wc_x, ca = wc_a, cb = wc_b, cz = wc_z;
        if constexpr (WALLS) {
            const int i = u - 3;
            if ((cx & kWallX) | (ca & kWallY) | (cb & kWallY) | (cz & (kWallZ | kWallSolid))) {
                const long long ib = (long long)i * PL;
                if (cx & kWallX) pf_x = ldg4(a.fr[0] + ib + PL + own);
                if (ca & kWallY) pf_y0 = ldg4(a.fr[1] + ib + (long long)jfa * sz + kb);
                if (cb & kWallY) pf_y1 = ldg4(a.fr[1] + ib + (long long)jfb * sz + kb);
                if (cz & kWallZ) pf_z = ldg4(a.fr[2] + ib + own);
                if (cz & kWallSolid) pf_s = __ldg(reinterpret_cast<const unsigned*>(a.solid + ib + own));
            }
            if (i >= i_beg && i < i_end) {
                if (a.fr[2] && h_ok) pf_h = __ldg(a.fr[2] + (long long)i * PL + (j0 + h_j) * sz + h_k);
                if (pl_node >= 0) {
                    const int node = pl_node + ny * i;
                    pl_c = __ldg(a.plate.code + node);
                    pl_w = __ldg(a.plate.w + node);
                    pl_wp = __ldg(a.plate.wp + node);
                }
                if (pl_halo) {
                    const int node = j0 + h_j + ny * i;
                    pl_hc = __ldg(a.plate.code + node);
                    pl_hw = __ldg(a.plate.w + node);
                    pl_hwp = __ldg(a.plate.wp + node);
                }
            }
            wc_z = wc_x;
            wall_codes(u + 1);
        }
        const bool ok = mbar_wait(bar0 + 8u * ps, (ph >> ps) & 1u, a.wait_us);
        // the source deposit, on the arriving plane's shared copy before anyone reads it
        if (u == dep_u && ok) {
            const float amp = a.dep_sig[a.dep_step];
            if (amp != 0.0f) {
                float* c = smem + C::RING0 + o0 + dep_at;
                *c = fadd(*c, amp);
            }
        }
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicMin(a.status + kStatusTimeout, blockIdx.x + gridDim.x * blockIdx.y);
            u_fail = u;
            return false;
        }
        ph ^= 1u << ps;
        // iteration u+D's loads go into the slots iteration u-1 freed (their last
        // reads came before the barrier above), so the issuing thread issues them
        // before its own work of this iteration rather than after it
        if (issuer && u + C::D <= u1) issue(u + C::D, ring(ps + C::D), vring(vs0 + C::D));
        float ax_next = 0.0f, px_next = 1.0f;
        if constexpr (!FAST) {
            ax_next = ax_at(u + 1);
            px_next = px_at(u - 2);
        }
        const float* vs = smem + C::VST0 + vs0 * C::V_STAGE;

        // ---- new Vx on face f = u-2 of the own columns (planes f-1 .. f+2) ----
        if (FAST || u >= i_beg) {
            const int f = u - 2, fg = f + xg0;
            float4 vnew = make_float4(0.f, 0.f, 0.f, 0.f);
            float4 vdiv = vnew;   // WALLS: the value the divergence sees
            if (FAST || (fg >= 0 && fg <= nxg - 2 && row_ok)) {   // rows beyond the room hold zeros
                const float4 pm = lds4(smem + C::RING0 + o3 + cP);
                const float4 p0 = lds4(smem + C::RING0 + o2 + cP);
                const float4 p1 = lds4(smem + C::RING0 + o1 + cP);
                const float4 p2 = lds4(smem + C::RING0 + o0 + cP);
                const float4 vo = lds4(vs + C::VX_OFF + 4 * tid);
                if constexpr (FAST) {
                    vnew = vel4(cf, pm, p0, p1, p2, vo, dxi);
                } else {
                    const bool fourth = (fg > 0 && fg < nxg - 2);
                    const float axf = axw2, axf1 = axw1;     // alpha_x[f], alpha_x[f+1]
                    if (fourth && axf == 0.0f && axf1 == 0.0f && kfull) {
                        vnew = vel4(cf, pm, p0, p1, p2, vo, dxi);
                    } else {
                        float4 aL, aR;
                        int okx = 0;
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            at(aL, q) = fmaxf(axf, at(myz, q));
                            at(aR, q) = fmaxf(axf1, at(myz, q));
                            okx |= (kb + q < nz) ? (1 << q) : 0;
                        }
                        vnew = vel4_general(cf, pm, p0, p1, p2, vo, aL, aR, fourth ? 15 : 0, okx);
                    }
                }
                if constexpr (WALLS) {
                    vdiv = vnew;
                    if (cx & kWallX) {
                        vnew = close4(vnew, pf_x);
                        vdiv = a.frac_div ? mul4(vnew, pf_x) : vnew;
                    }
                }
                if (f >= i_beg && f < i_end && st_ok) {
                    if constexpr (FAST) stg4(gX, vnew);
                    else stg4(a.vout[0] + f * PL + own, vnew);
#pragma unroll
                    for (int sd = 0; sd < 2; ++sd)   // the neighbours' ghost faces
                        if (PEER && a.pr.vx[sd] && f >= a.pr.v_lo[sd] && f < a.pr.v_hi[sd])
                            stg4(a.pr.vx[sd] + (f + a.pr.dl[sd]) * PL + own, vnew);
                }
            }
            qx0 = qx1; qx1 = qx2; qx2 = qx3; qx3 = WALLS ? vdiv : vnew;
        }

        // ---- plane i = u-3: new Vy / Vz (with halos), then P^{n+1} ----
        {
            const int i = u - 3;
            if (FAST || i >= i_beg) {
                const float axi = FAST ? 0.0f : axw3;    // alpha_x[i]
                const bool xint = FAST || (axi == 0.0f);
                const float* pst = smem + C::RING0 + o3;
                const float* vys = vs + C::VY_OFF;
                const float* vzs = vs + C::VZ_OFF;
                const long long ib = i * PL;

                // Vy rows: row w, and row TJ+w for the first VYR-TJ warps
                if constexpr (FAST) {
                    const float* pc = pst + 4 * lane + 4;
                    auto row = [&](int r, const float4& dmp, bool ex, bool f4, float4 fry, unsigned c, float* dst) {
                        const float4 pm = lds4(pc + r * C::PC), p0 = lds4(pc + (r + 1) * C::PC);
                        const float4 p1 = lds4(pc + (r + 2) * C::PC), p2 = lds4(pc + (r + 3) * C::PC);
                        const float4 vo = lds4(vys + r * C::TK + 4 * lane);
                        float4 v;
                        if (jmid) v = vel4(cf, pm, p0, p1, p2, vo, dmp);
                        else v = vel4_masked(cf, pm, p0, p1, p2, vo, dmp, f4 ? 15 : 0, ex ? 15 : 0);
                        if constexpr (WALLS) {
                            if (c & kWallY) v = close4(v, fry);
                        }
                        if (dst) stg4(dst, v);
                        if constexpr (WALLS) {
                            if ((c & kWallY) && a.frac_div) v = mul4(v, fry);
                        }
                        sts4(vyn + r * C::TK + 4 * lane, v);
                    };
                    // own rows are r = 2 .. TJ+1 of the tile's Vy rows
                    row(w, dyi[0], ya_ok, ya_4, pf_y0, ca, w >= 2 && ya_ok && kb < sz ? gYa : nullptr);
                    if (C::TJ + w < C::VYR)
                        row(C::TJ + w, dyi[1], yb_ok, yb_4, pf_y1, cb, w < 2 && yb_ok && kb < sz ? gYb : nullptr);
                } else {
#pragma unroll
                    for (int m = 0; m < NY_IT; ++m) {
                        const int r = m == 0 ? w : C::TJ + w;
                        if (r < C::VYR) {
                            const int jf = j0 - 2 + r;
                            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                            if (jf >= 0 && jf <= ny - 2) {
                                const float* pc = pst + 4 * lane + 4;
                                const float4 pm = lds4(pc + r * C::PC), p0 = lds4(pc + (r + 1) * C::PC);
                                const float4 p1 = lds4(pc + (r + 2) * C::PC), p2 = lds4(pc + (r + 3) * C::PC);
                                const float4 vo = lds4(vys + r * C::TK + 4 * lane);
                                {
                                    const bool fourth = (jf > 0 && jf < ny - 2);
                                    if (fourth && xint && kfull) {
                                        v = vel4(cf, pm, p0, p1, p2, vo, dyi[m]);
                                    } else {
                                        float4 aL, aR;
                                        int oky = 0;
#pragma unroll
                                        for (int q = 0; q < 4; ++q) {
                                            const float azk = az_s[4 * lane + 4 + q];
                                            at(aL, q) = fmaxf(fmaxf(axi, ay_s[r]), azk);
                                            at(aR, q) = fmaxf(fmaxf(axi, ay_s[r + 1]), azk);
                                            oky |= (kb + q < nz) ? (1 << q) : 0;
                                        }
                                        v = vel4_general(cf, pm, p0, p1, p2, vo, aL, aR, fourth ? 15 : 0, oky);
                                    }
                                }
                                float4 fry = make_float4(1.f, 1.f, 1.f, 1.f);
                                if constexpr (WALLS) {
                                    if ((m == 0 ? ca : cb) & kWallY) {
                                        fry = m == 0 ? pf_y0 : pf_y1;
                                        v = close4(v, fry);
                                    }
                                }
                                if (r >= 2 && r < C::TJ + 2 && kb < sz)
                                    stg4(a.vout[1] + ib + (long long)jf * sz + kb, v);
                                if constexpr (WALLS) {
                                    if (((m == 0 ? ca : cb) & kWallY) && a.frac_div) v = mul4(v, fry);
                                }
                            }
                            sts4(vyn + r * C::TK + 4 * lane, v);
                        }
                    }

                }

                // Vz: own faces kb .. kb+3 of row jr
                float4 pown = make_float4(0.f, 0.f, 0.f, 0.f);
                {
                    const float* prow = pst + (w + 3) * C::PC;
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (FAST || row_ok) {
                        const int c = 4 * lane + 4;            // col of kb
                        pown = lds4(prow + c);
                        const float4 pb4 = lds4(prow + c + 4);
                        const float pl = prow[c - 1];
                        const float4 vo = lds4(vzs + w * C::PC + c);
                        // faces kb+q use P[kb+q-1 .. kb+q+2]
                        const float4 pm = make_float4(pl, pown.x, pown.y, pown.z);
                        const float4 p1 = make_float4(pown.y, pown.z, pown.w, pb4.x);
                        const float4 p2 = make_float4(pown.z, pown.w, pb4.x, pb4.y);
                        if (xint) {
                            v = vel4_masked(cf, pm, pown, p1, p2, vo, dzi, zm4, zok);
                        } else {
                            const float ay = ay_s[w + 2];
                            float4 aL, aR;
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                at(aL, q) = fmaxf(fmaxf(axi, ay), az_s[c + q]);
                                at(aR, q) = fmaxf(fmaxf(axi, ay), az_s[c + q + 1]);
                            }
                            v = vel4_general(cf, pm, pown, p1, p2, vo, aL, aR, zm4, zok);
                        }
                        float4 frz = make_float4(1.f, 1.f, 1.f, 1.f);
                        if constexpr (WALLS) {
                            if (cz & kWallZ) {
                                frz = pf_z;
                                v = close4(v, frz);
                            }
                            if (pl_c) {
                                const float vp = fmul(fsub(pl_w, pl_wp), a.plate.inv_dt);
#pragma unroll
                                for (int q = 0; q < 4; ++q) at(v, q) = plate_face(at(v, q), kb + q, pl_c, vp);
                            }
                        }
                        if (st_ok) stg4(FAST ? gZ : a.vout[2] + ib + own, v);
                        if constexpr (WALLS) {
                            if ((cz & kWallZ) && a.frac_div) v = mul4(v, frz);
                        }
                    }
                    sts4(vzn + w * C::PC + 4 * lane + 4, v);
                }
                // halo Vz faces k0-2, k0-1, k0+TK of every row: 3*TJ faces, one per
                // thread of the last HW warps
                if (h_mine) {
                    const float* pr = pst + h_p;
                    float vh = 0.0f;
                    if (h_ok) {
                        const float gr = grad4(cf, pr[-1], pr[0], pr[1], pr[2], h_4);
                        float dmp = h_d;
                        if constexpr (!FAST) {
                            const float mxy = fmaxf(axi, ay_s[h_j + 2]);
                            dmp = face_damp(fmaxf(mxy, az_s[h_c]), fmaxf(mxy, az_s[h_c + 1]), cf.dt);
                        }
                        vh = vupd(cf, vzs[h_v], gr, dmp);
                        if constexpr (WALLS) {
                            if (pf_h == 0.0f) vh = 0.0f;   // 1 without fractions
                            if (pl_hc) vh = plate_face(vh, h_k, pl_hc, fmul(fsub(pl_hw, pl_hwp), a.plate.inv_dt));
                            if (a.frac_div) vh = fmul(vh, pf_h);
                        }
                    }
                    vzn[h_v] = vh;
                }
                __syncthreads();

                // P^{n+1} of the own cells
                if (FAST || row_ok) {
                    const float* yr = vyn + 4 * lane;
                    const float4 ymm = lds4(yr + w * C::TK), ym = lds4(yr + (w + 1) * C::TK);
                    const float4 yp = lds4(yr + (w + 2) * C::TK), ypp = lds4(yr + (w + 3) * C::TK);
                    const float* zr = vzn + w * C::PC + 4 * lane;
                    const float2 za = *reinterpret_cast<const float2*>(zr + 2);   // faces kb-2, kb-1
                    const float4 zb = lds4(zr + 4);                                // faces kb .. kb+3
                    const float zc = zr[8];                                        // face kb+4
                    // px[i] = 1 on x-interior planes, so min(px[i], min(py, pz)) = mpz there
                    float4 pd = mpz;
                    if constexpr (!FAST) {
                        const float pxi = pxw;
#pragma unroll
                        for (int q = 0; q < 4; ++q) at(pd, q) = fminf(pxi, at(mpz, q));
                    }
                    float4 out;
                    out.x = pupd(cf, pown.x, qx2.x, qx1.x, qx3.x, qx0.x, yp.x, ym.x, ypp.x, ymm.x, zb.x, za.y, zb.y, za.x, pd.x);
                    out.y = pupd(cf, pown.y, qx2.y, qx1.y, qx3.y, qx0.y, yp.y, ym.y, ypp.y, ymm.y, zb.y, zb.x, zb.z, za.y, pd.y);
                    out.z = pupd(cf, pown.z, qx2.z, qx1.z, qx3.z, qx0.z, yp.z, ym.z, ypp.z, ymm.z, zb.z, zb.y, zb.w, zb.x, pd.z);
                    out.w = pupd(cf, pown.w, qx2.w, qx1.w, qx3.w, qx0.w, yp.w, ym.w, ypp.w, ymm.w, zb.w, zb.z, zc, zb.y, pd.w);
                    if (!kfull) {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (kb + q >= nz) at(out, q) = 0.0f;
                    }
                    if constexpr (WALLS) {
                        if (cz & kWallSolid) {   // solid cells keep P = 0
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                if ((pf_s >> (8 * q)) & 0xFFu) at(out, q) = 0.0f;
                        }
                    }
                    if (FAST ? st_ok : kb < sz) {
                        stg4(FAST ? gP : a.pn + ib + own, out);
#pragma unroll
                        for (int sd = 0; sd < 2; ++sd)   // the neighbours' ghost planes
                            if (PEER && a.pr.pn[sd] && i >= a.pr.p_lo[sd] && i < a.pr.p_hi[sd])
                                stg4(a.pr.pn[sd] + (i + a.pr.dl[sd]) * PL + own, out);
                    }
                }
            }
        }

        if constexpr (!FAST) {
            axw3 = axw2; axw2 = axw1; axw1 = axw0; axw0 = ax_next;
            pxw = px_next;
        }
        ps = ring(ps + 1);
        vs0 = vring(vs0 + 1);
        o3 = o2; o2 = o1; o1 = o0;
        o0 = ps * C::P_STAGE;
        if constexpr (FAST) {
            gX += PL; gYa += PL; gYb += PL; gZ += PL; gP += PL;
        }
        return true;
    };

    for (int u = u0; u <= u1;) {
        if (u == fast_lo) {
            bool ran = true;
            const long long ib = (long long)(u - 3) * PL;
            gX = a.vout[0] + ib + PL + own;
            gYa = a.vout[1] + ib + (long long)jfa * sz + kb;
            gYb = a.vout[1] + ib + (long long)jfb * sz + kb;
            gZ = a.vout[2] + ib + own;
            gP = a.pn + ib + own;
            for (; u < fast_hi; ++u)
                if (!iteration(u, std::true_type{})) { ran = false; break; }
            if (!ran) break;
            // the window of the general iterations that follow
            axw3 = ax_at(u - 3); axw2 = ax_at(u - 2); axw1 = ax_at(u - 1); axw0 = ax_at(u);
            pxw = px_at(u - 3);
            continue;
        }
        if (!iteration(u, std::false_type{})) break;
        ++u;
    }

    pp.ps = ps;
    pp.vs = vs0;
    pp.ph = ph;
    // A normal march waits for every load it issued, so none is in flight here.
    // After a timed-out wait at iteration u_fail, the copies issued for
    // iterations u_fail .. u_fail+D-1 may still be landing: wait for them
    // (bounded) before the CTA's shared memory is released.
    if (u_fail <= u1) {
        if (tid == 0) {
            for (int q = 0; q < C::D && u_fail + q <= u1; ++q) {
                const int sl = ring(ps + q);
                mbar_wait(bar0 + 8u * sl, (ph >> sl) & 1u, a.wait_us);
            }
        }
        __syncthreads();
        return false;
    }
    return true;
}

// Single-room step: one CTA per (tile, segment).
template <class C, bool PEER, bool WALLS = false>
__global__ void __launch_bounds__(C::NT) k_fused_step(FusedArgs a,
                                                      const __grid_constant__ CUtensorMap tmP,
                                                      const __grid_constant__ CUtensorMap tmX,
                                                      const __grid_constant__ CUtensorMap tmY,
                                                      const __grid_constant__ CUtensorMap tmZ,
                                                      int seg_len, int tiles_k)
{
    if ((int)blockIdx.y * seg_len >= (a.xs.nxg > 0 ? a.xs.n_own : a.g.nx)) return;
    if constexpr (WALLS) {
        if (a.gate && a.gate[kStatusPlate] != 0xFFFFFFFFu) return;
    }
    float* smem;
    const unsigned sbase = smem_base_u32<C>(&smem);
    const unsigned bar0 = sbase + 4u * C::BAR0;
    init_barriers<C>(bar0);
    Pipe pp;
    fused_tile<C, PEER, WALLS>(a, &tmP, &tmX, &tmY, &tmZ, blockIdx.x, blockIdx.y * seg_len, seg_len, tiles_k, smem,
                               sbase, bar0, pp, [&] {
        return [&] {
            // the previous step's receivers, from this step's input P
            const int nblk = gridDim.x * gridDim.y, b = blockIdx.x + gridDim.x * blockIdx.y;
            for (int r = b + nblk * (int)threadIdx.x; r < a.n_rec; r += nblk * C::NT)
                a.rec_out[r] = sample8(a.p, a.rec_idx + 8 * r, a.rec_w + 8 * r);
        };
    });
}

// Batched step: a persistent kernel whose CTAs pull (member, tile, segment)
// work items from a device counter until the list is exhausted; members at
// their step limit are skipped.  Uneven members balance across the SMs.  The
// members' tensor maps live in global memory and are rewritten when the set
// changes, so each work item acquires them before its first TMA load.
template <class C>
__global__ void __launch_bounds__(C::NT, 2) k_fused_batch(BatchMember* __restrict__ mem,
                                                          BatchHeader* __restrict__ hdr,
                                                          const int4* __restrict__ items,
                                                          unsigned* __restrict__ status)
{
    __shared__ int s_item;
    float* smem;
    const unsigned sbase = smem_base_u32<C>(&smem);
    const unsigned bar0 = sbase + 4u * C::BAR0;
    init_barriers<C>(bar0);
    Pipe pp;
    wait_previous();
    release_next();
    const int total_items = hdr->total_items;
    int* const counter = &hdr->counter;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        const int item = s_item;
        __syncthreads();
        if (item >= total_items) break;
        const int4 it = items[item];   // member, tile, first plane, planes
        const BatchMember* m = mem + it.x;
        const int step = m->step;
        if (step >= m->limit || m->unstable != 0xFFFFFFFFu) continue;   // done, or stopped unstable
        const int par = (step - m->step0) & 1;
        FusedArgs a;
        a.g = m->g;
        a.cf = m->cf;
        a.tb = m->tb;
        a.p = m->p[par];
        a.pn = m->p[par ^ 1];
        for (int c = 0; c < 3; ++c) {
            a.vin[c] = m->v[par][c];
            a.vout[c] = m->v[par ^ 1][c];
        }
        a.status = status;
        a.xs = XSpan{0, 0, 0, 0};
        a.pr = XPeers{};
        if (!fused_tile<C, false>(a, &m->maps[par][0], &m->maps[par][1], &m->maps[par][2], &m->maps[par][3],
                           it.y, it.z, it.w, m->tiles_k, smem, sbase, bar0, pp, [&] {
            if (threadIdx.x == C::NT / 2)   // the thread that issues the loads
                for (int q = 0; q < 4; ++q) acquire_tensormap(&m->maps[par][q]);
            return [] {};
        }))
            break;
    }
}

// After a batched step, per member below its limit: record the receivers from
// the new pressure, advance the step counter, run the 256-step check, then
// deposit the next step's source sample (the order of the single-room path:
// record after step n, deposit before step n+1).  One block per member.  A
// member whose check fails stops at that step without the next deposit, the
// state a single room is left in when its step returns UNSTABLE; the batch
// steps it no further until its set is rebuilt.  The first block also returns
// the work-item counter to zero for the next step.
__global__ void __launch_bounds__(128) k_batch_epilogue(BatchMember* __restrict__ mem, BatchHeader* __restrict__ hdr)
{
    const int r = blockIdx.x;
    const bool in = r < hdr->n_members;
    BatchMember* m = mem + r;
    // a member's description does not change between steps: fetch it, and the
    // taps of this thread's receiver, while the step's last tiles finish
    float *p0 = nullptr, *p1 = nullptr, *trace = nullptr, w[8];
    long long idx[8];
    int n_rec = 0, step0 = 0, limit = 0, trace0 = 0, trace_cap = 0;
    if (in) {
        p0 = m->p[0];
        p1 = m->p[1];
        trace = m->trace;
        n_rec = m->n_rec;
        step0 = m->step0;
        limit = m->limit;
        trace0 = m->trace0;
        trace_cap = m->trace_cap;
        if ((int)threadIdx.x < n_rec)
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                idx[t] = m->rec_idx[8 * threadIdx.x + t];
                w[t] = m->rec_w[8 * threadIdx.x + t];
            }
    }
    wait_previous();
    release_next();
    if (r == 0 && threadIdx.x == 0) hdr->counter = 0;
    if (!in) return;
    const int s = *(volatile int*)&m->step;
    if (s >= limit || *(volatile unsigned*)&m->unstable != 0xFFFFFFFFu) return;
    const int s1 = s + 1;
    float* P = ((s1 - step0) & 1) ? p1 : p0;
    const int slot = trace0 + (s - step0);
    if (slot < trace_cap)
        for (int q = threadIdx.x; q < n_rec; q += blockDim.x)
            trace[(size_t)slot * n_rec + q] =
                q < (int)blockDim.x ? sample8(P, idx, w) : sample8(P, m->rec_idx + 8 * q, m->rec_w + 8 * q);
    if ((s1 & (kCheckPeriod - 1)) == 0) {
        const int n_chk = s1 / kCheckPeriod - step0 / kCheckPeriod;
        const long long phase = (m->phase0 + n_chk - 1) % kCheckStride;
        const Grid g = m->g;
        for (long long q = phase + (long long)kCheckStride * threadIdx.x; q < m->n_cells;
             q += (long long)kCheckStride * blockDim.x) {
            const int k = (int)(q % g.nz);
            const long long ij = q / g.nz;
            const float v = P[((ij / g.ny) * g.ny + ij % g.ny) * g.sz + k];
            if (!isfinite(v) || v > 2e3f || v < -2e3f) atomicCAS(&m->unstable, 0xFFFFFFFFu, (unsigned)s1);
        }
    }
    __syncthreads();   // receivers have read P and the check's flags are set
    if (threadIdx.x == 0) {
        const bool stopped = *(volatile unsigned*)&m->unstable != 0xFFFFFFFFu;
        if (!stopped && s1 < limit && s1 < m->ps_n) deposit_apply(m->ps, m->ps_sig[s1], P);
        m->step = s1;
    }
}

using FusedCfg = Cfg<8, 2>;          // 8 x 128 tiles: single rooms, and batches by default
using NarrowCfg = Cfg<16, 2, 16>;    // 16 x 64 tiles: batches of rooms with small Nz

constexpr int kMaxDevices = 64;
int g_slots_per_sm[2][kMaxDevices];   // per tile shape and device
int g_sms[2][kMaxDevices];
bool g_configured[2][kMaxDevices];

}  // namespace

namespace {
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::once_flag g_encode_once;

cudaError_t get_encoder()
{
    std::call_once(g_encode_once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    });
    return g_encode ? cudaSuccess : cudaErrorNotSupported;
}
}  // namespace

cudaError_t encode_field_map(CUtensorMap* m, const void* base, int elem_bytes, const Grid& g, int bx, int by)
{
    cudaError_t e = get_encoder();
    if (e != cudaSuccess) return e;
    if (elem_bytes != 4 && elem_bytes != 2) return cudaErrorInvalidValue;
    const cuuint64_t eb = (cuuint64_t)elem_bytes;
    cuuint64_t dims[3] = {(cuuint64_t)g.sz, (cuuint64_t)g.ny, (cuuint64_t)g.nx};
    cuuint64_t strides[2] = {(cuuint64_t)g.sz * eb, (cuuint64_t)g.plane * eb};
    cuuint32_t box[3] = {(cuuint32_t)bx, (cuuint32_t)by, 1};
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = g_encode(m, elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 3,
                          const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

struct FusedCache {
    struct Entry {
        const float* base;
        int kind, shape;
        CUtensorMap map;
    };
    std::vector<Entry> entries;
};

FusedCache* fused_cache_create() { return new FusedCache(); }
void fused_cache_destroy(FusedCache* c) { delete c; }

template <class C>
void box_of(int kind, int* bx, int* by)
{
    const int x[4] = {C::PC, C::TK, C::TK, C::PC};
    const int y[4] = {C::PR, C::TJ, C::VYR, C::TJ};
    *bx = x[kind];
    *by = y[kind];
}

static cudaError_t cached_map(FusedCache* c, const float* base, int kind, const Grid& g, CUtensorMap* out,
                              int shape = 0)
{
    for (const auto& e : c->entries)
        if (e.base == base && e.kind == kind && e.shape == shape) { *out = e.map; return cudaSuccess; }
    int bx, by;
    if (shape == 1) box_of<NarrowCfg>(kind, &bx, &by);
    else box_of<FusedCfg>(kind, &bx, &by);
    FusedCache::Entry e;
    e.base = base;
    e.kind = kind;
    e.shape = shape;
    cudaError_t err = encode_field_map(&e.map, base, 4, g, bx, by);
    if (err != cudaSuccess) return err;
    c->entries.push_back(e);
    *out = e.map;
    return cudaSuccess;
}

bool fused_supported(const Grid& g)
{
    return g.nx >= 1 && g.ny >= 1 && g.nz >= 1 && (g.sz % 8) == 0;
}

int fused_kernel_launches_per_step() { return 1; }

template <class C>
static cudaError_t launch_step_of(const FusedArgs& a, FusedCache* cache, cudaStream_t s, int shape)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    if (!g_configured[shape][dev]) {
        e = cudaFuncSetAttribute(k_fused_step<C, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)C::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        e = cudaFuncSetAttribute(k_fused_step<C, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)C::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        e = cudaFuncSetAttribute(k_fused_step<C, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)C::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        e = cudaDeviceGetAttribute(&g_sms[shape][dev], cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        int slots = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&slots, k_fused_step<C, true>, C::NT, C::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        int slots_w = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&slots_w, k_fused_step<C, false, true>, C::NT,
                                                          C::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        slots = slots < slots_w ? slots : slots_w;
        g_slots_per_sm[shape][dev] = slots > 0 ? slots : 1;
        g_configured[shape][dev] = true;
    }
    const Grid& g = a.g;
    CUtensorMap maps[4];
    const float* bases[4] = {a.p, a.vin[0], a.vin[1], a.vin[2]};
    for (int q = 0; q < 4; ++q) {
        e = cached_map(cache, bases[q], q, g, &maps[q], shape);
        if (e != cudaSuccess) return e;
    }
    const int tiles_j = (g.ny + C::TJ - 1) / C::TJ;
    const int tiles_k = (g.nz + C::TK - 1) / C::TK;
    const long long tiles = (long long)tiles_j * tiles_k;
    // segments along i: as many as one wave of resident CTAs holds (every CTA
    // marches the same number of planes, so a single full wave has no tail)
    const long long slots = (long long)g_slots_per_sm[shape][dev] * g_sms[shape][dev];
    const int n_own = a.xs.nxg > 0 ? a.xs.n_own : g.nx;
    long long segs = slots / tiles;
    if (segs < 1) segs = 1;
    if (segs > n_own) segs = n_own;
    const int seg_len = (int)((n_own + segs - 1) / segs);
    segs = (n_own + seg_len - 1) / seg_len;
    dim3 grid((unsigned)tiles, (unsigned)segs, 1);
    const bool peer = a.pr.pn[0] || a.pr.pn[1] || a.pr.vx[0] || a.pr.vx[1];
    const bool walls = a.fr[0] || a.fr[1] || a.fr[2] || a.solid || a.plate.code;
    if (walls && (peer || a.xs.nxg > 0)) return cudaErrorInvalidValue;   // walled scenes are whole rooms
    // Plain launches: overlapping a step's start with the one before (launch.h)
    // was slower (512x384x256 room 266.6 -> 281 us, 160x128x112 24.7 -> 25.4).
    if (walls)
        k_fused_step<C, false, true><<<grid, C::NT, C::SMEM_BYTES, s>>>(a, maps[0], maps[1], maps[2], maps[3],
                                                                        seg_len, tiles_k);
    else if (peer)
        k_fused_step<C, true><<<grid, C::NT, C::SMEM_BYTES, s>>>(a, maps[0], maps[1], maps[2], maps[3], seg_len,
                                                                 tiles_k);
    else
        k_fused_step<C, false><<<grid, C::NT, C::SMEM_BYTES, s>>>(a, maps[0], maps[1], maps[2], maps[3], seg_len,
                                                                  tiles_k);
    return cudaGetLastError();
}

// The tile shape a room's step uses: 16 x 64 tiles when they leave less of the
// last k tile idle than 8 x 128 tiles (e.g. Nz = 32, 48, 144, 160), else 8 x 128.
int fused_step_shape(const Grid& g)
{
    const int w128 = (g.nz + 127) / 128 * 128 - g.nz, w64 = (g.nz + 63) / 64 * 64 - g.nz;
    return w64 < w128 ? 1 : 0;
}

cudaError_t launch_fused_step(const FusedArgs& a, FusedCache* cache, cudaStream_t s)
{
    return fused_step_shape(a.g) == 1 ? launch_step_of<NarrowCfg>(a, cache, s, 1)
                                      : launch_step_of<FusedCfg>(a, cache, s, 0);
}

cudaError_t fused_maps(FusedCache* c, const Grid& g, const float* p, const float* const* v,
                       CUtensorMap out[4], int shape)
{
    const float* bases[4] = {p, v[0], v[1], v[2]};
    for (int q = 0; q < 4; ++q) {
        cudaError_t e = cached_map(c, bases[q], q, g, &out[q], shape);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void fused_tile_shape(int shape, int* tj, int* tk)
{
    *tj = shape == 1 ? NarrowCfg::TJ : FusedCfg::TJ;
    *tk = shape == 1 ? NarrowCfg::TK : FusedCfg::TK;
}

template <class C>
static cudaError_t batch_slots_of(int* slots)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_fused_batch<C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    int sms = 0, per = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_fused_batch<C>, C::NT, C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    *slots = (per > 0 ? per : 1) * sms;
    return cudaSuccess;
}

cudaError_t fused_batch_slots(int shape, int* slots)
{
    return shape == 1 ? batch_slots_of<NarrowCfg>(slots) : batch_slots_of<FusedCfg>(slots);
}

cudaError_t launch_fused_batch_step(BatchMember* members, BatchHeader* hdr, const int4* items,
                                    unsigned* status, int grid_ctas, int epi_blocks, cudaStream_t s,
                                    int shape)
{
    cudaError_t e;
    if (shape == 1)
        e = launch_after(k_fused_batch<NarrowCfg>, dim3(grid_ctas), dim3(NarrowCfg::NT), NarrowCfg::SMEM_BYTES, s, members,
                         hdr, items, status);
    else
        e = launch_after(k_fused_batch<FusedCfg>, dim3(grid_ctas), dim3(FusedCfg::NT), FusedCfg::SMEM_BYTES, s, members,
                         hdr, items, status);
    if (e != cudaSuccess) return e;
    return launch_after(k_batch_epilogue, dim3(epi_blocks), dim3(128), 0, s, members, hdr);
}

}  // namespace fdtd
