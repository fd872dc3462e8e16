// FP32 form, 3D uniform grids: TMA-tiled fused stage kernels.
//
// A CTA owns a TX x TY (x, y) column of cells and marches a chunk of kc
// z-planes.  Each plane of the stage input is staged once into shared memory
// by one TMA box copy ((TX+8) x (TY+6) floats: the tile plus its 3-cell x/y
// halo, x rounded down to a 16-byte boundary) into a ring of RING slots
// guarded by mbarriers; the ring holds the seven planes of the z stencil as
// well as the planes being prefetched.  Every thread computes two
// x-adjacent cells in each of RY consecutive rows with packed FP32x2
// arithmetic (Blackwell FFMA2/FADD2/FMUL2); the rows of a thread are
// independent chains of arithmetic and share their y-stencil loads.  The
// WENO5-HJ upwind side and the Godunov branch of the reinitialisation are
// chosen with selects: the plus-side derivative is the minus-side formula on
// the mirrored difference sequence, so one evaluation per axis serves both
// sides.  The tile shape, the rows per thread and the ring depth form a
// configuration (TileCfg, kTileCfgs); the autotuner picks one per size
// class, with the z chunk.
//
// Waits on the mbarriers are bounded: on a timeout the kernel raises the
// instance's error flag, waits (bounded) for its copies in flight and
// returns; the host reports R3D_ETIMEOUT.
#include <cuda.h>

#include <string>

#include "stencil_f32.cuh"
#include "tile_host.h"

namespace r3d {

namespace {

constexpr long long kSpin = 1ll << 22;

// ------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, long long limit = kSpin) {
    for (long long it = 0; it < limit; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// plain tiled TMA load of one box into this CTA's own shared memory
__device__ __forceinline__ void tma_load_3d(float* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// ------------------------------------------------------------ packed math
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(rcp_approx(a.x), rcp_approx(a.y)); }
__device__ __forceinline__ float2 sel2(bool cx, bool cy, float2 a, float2 b) {
    return make_float2(cx ? a.x : b.x, cy ? a.y : b.y);
}

// WENO5 (Jiang-Peng) on a uniform axis, twice the derivative times h, as the
// central difference M = f[+1] - f[-1] less a correction of the second
// differences E_j = f[j+1] - 2 f[j] + f[j-1] around the cell.  With
//   a, b, c, d = E_-2, E_-1, E_0, E_+1   (minus side; the plus side mirrors
//   the axis: E_+2, E_+1, E_0, E_-1, and the correction changes its sign)
// the three smoothness indicators plus psi = 1e-6, times h^2 and over their
// leading coefficients, are sums of squares,
//   s1 = (c - 0.55 d)^2 + 0.0975 d^2 + 0.3e-6 h^2      (IS1 10/3 of it)
//   s2 = (b - 0.625 c)^2 + 0.609375 c^2 + 0.75e-6 h^2  (IS2  4/3 of it)
//   s3 = (b - 0.55 a)^2 + 0.0975 a^2 + 0.3e-6 h^2      (IS3 10/3 of it)
// and the weights w_r = (c_r/s_r^2) / sum enter through the ratios p = s1/s2,
// q = s3/s2: with P = p^2, Q = 1.5 q^2 the correction is
//   (1/3) [ c - b + (P (a-2b+c) + Q (b-2c+d)) / (P/2 + Q + 12.5 P Q) ].
// Ratios need no scaling against the FP32 range whatever h is.  One of p, q
// is always above 0.05 (s1 >= 0.24 c^2, s3 >= 0.24 b^2, s2 <= 2 (b^2 + c^2)
// plus the psi terms), so the denominator cannot vanish; 1e-15 (s1 + s3)
// added to s2 bounds the ratios by 1e15, so that P and Q stay in range.  A
// denominator that leaves it (P Q above 2.7e37) gives F, off by weights below
// 1e-8.  The range ends where a second difference squared does, at 1e19 (1e16
// and up in the reinitialisation, which squares gradients too): not finite
// there.  The error is 2^-24 of the largest second difference in the stencil,
// spikes of any size included; the form with three products of squared
// indicators, clamped at 1e6, was off by half a spike's size from 10 up and not
// finite from 1e16 on.
// 31 packed operations and no clamps after the selects, where the form with
// three products of squared indicators took 37 and 6, and half the distinct
// constants (the registers that hold them limit the CTAs per SM).  With the
// plane loop's address and wall-ghost arithmetic cut at the same time, the
// 256^3 stages went 140 -> 121 us (convection, 397 -> ~340 warp instructions
// per 64 cells; issue-bound) and 187 -> 133 us (reinitialisation of five
// spheres, most of it the interface band below).
__device__ __forceinline__ float2 weno5_corr(float2 a, float2 b, float2 c, float2 d, float psi1, float psi2) {
    const float2 x1 = fma2(f2(-0.55f), d, c), x2 = fma2(f2(-0.625f), c, b), x3 = fma2(f2(-0.55f), a, b);
    const float2 s1 = fma2(x1, x1, fma2(mul2(f2(0.0975f), d), d, f2(psi1)));
    const float2 s2 = fma2(x2, x2, fma2(mul2(f2(0.609375f), c), c, f2(psi2)));
    const float2 s3 = fma2(x3, x3, fma2(mul2(f2(0.0975f), a), a, f2(psi1)));
    const float2 rho = rcp2(fma2(f2(1.0e-15f), add2(s1, s3), s2));
    const float2 p = mul2(s1, rho), q = mul2(s3, rho);
    const float2 P = mul2(p, p), Q = mul2(mul2(f2(1.5f), q), q);
    const float2 inv = rcp2(fma2(P, fma2(Q, f2(12.5f), f2(0.5f)), Q));
    const float2 F = sub2(c, b);
    const float2 G0 = add2(sub2(a, b), F), G2 = sub2(sub2(d, c), F);
    return fma2(fma2(P, G0, mul2(Q, G2)), inv, F);
}

// Twice the upwind derivative times h of an axis from its second differences
// e[0..4] (cells -2..+2) and the central difference m; plus side where px, py.
__device__ __forceinline__ float2 deriv2(const float2* e, float2 m, bool px, bool py, float psi1, float psi2) {
    const float2 r = weno5_corr(sel2(px, py, e[4], e[0]), sel2(px, py, e[3], e[1]), e[2], sel2(px, py, e[1], e[3]),
                                psi1, psi2);
    constexpr float third = 1.0f / 3.0f;
    return fma2(make_float2(px ? third : -third, py ? third : -third), r, m);
}

// WENO5 (Jiang-Peng) derivative times h in FP64 from the undivided
// differences d1..d5 of the minus-side upwind set (the plus side passes the
// mirrored set), the weights with one division:
// w_r = c_r prod_{q!=r} s_q^2 / sum_q c_q prod_{p!=q} s_p^2.
__device__ __forceinline__ double weno5_d(double d1, double d2, double d3, double d4, double d5, double eps) {
    const double a1 = d3 - d4, b1 = d5 - d4, b2 = d2 - d3, b3 = d1 - d2;
    const double s1 = ((10.0 / 3.0) * a1 + (11.0 / 3.0) * b1) * a1 + (4.0 / 3.0) * b1 * b1 + eps;
    const double s2 = ((4.0 / 3.0) * a1 - (5.0 / 3.0) * b2) * a1 + (4.0 / 3.0) * b2 * b2 + eps;
    const double s3 = ((10.0 / 3.0) * b2 - (11.0 / 3.0) * b3) * b2 + (4.0 / 3.0) * b3 * b3 + eps;
    const double q1 = s1 * s1, q2 = s2 * s2, q3 = s3 * s3;
    const double n1 = 0.3 * q2 * q3, n2 = 0.6 * q1 * q3, n3 = 0.1 * q1 * q2;
    const double p1 = d4 + (1.0 / 3.0) * a1 - (1.0 / 6.0) * b1;
    const double p2 = d3 - (1.0 / 3.0) * a1 - (1.0 / 6.0) * b2;
    const double p3 = d2 + (1.0 / 3.0) * b3 - (11.0 / 6.0) * b2;
    return (n1 * p1 + n2 * p2 + n3 * p3) / (n1 + n2 + n3);
}

// The interface band of the reinitialisation in FP64: the Godunov selection
// and one-sided WENO5 of one axis (src/reinidisc_f.cpp:70-109 on a uniform
// grid), squared, from the FP32 7-point stencil of the axis (centre f3): rh
// the FP32 1/h, eps = 1e-6 h^2 with h = 1/(double)rh (host-made).
__device__ __noinline__ double band_axis(float f0, float f1, float f2_, float f3, float f4, float f5, float f6,
                                         float rh, double eps) {
    const double sg = fabs((double)f3) < 1.0e-8 ? 1.0 : (f3 > 0.f ? 1.0 : -1.0);
    const double D2 = (double)f3 - (double)f2_, D3 = (double)f4 - (double)f3;
    const double ms = D2 * sg, ps = D3 * sg, sum = ms + ps;
    const bool c1 = ms > 0.0 && sum > 0.0, c2 = ps < 0.0 && sum < 0.0;
    if (!(c1 || c2)) return 0.0;
    const double D0 = (double)f1 - (double)f0, D1 = (double)f2_ - (double)f1;
    const double D4 = (double)f5 - (double)f4, D5 = (double)f6 - (double)f5;
    const double w = weno5_d(c2 ? D5 : D0, c2 ? D4 : D1, c2 ? D3 : D2, c2 ? D2 : D3, c2 ? D1 : D4, eps);
    const double gd = w * (double)rh;
    return gd * gd;
}

// The right-hand side -(S |grad| - S) of a band cell of value f0 from the
// squared gradient, with the smoothed sign of src/reinidisc_f.cpp:111-127.
__device__ __forceinline__ float band_rhs(float f0f, double g2, float deltax) {
    const double f0 = f0f, dl = deltax;
    const double dn = sqrt(g2);
    const double x = f0 * f0 + g2 * dl * dl;
    // f0 / sqrt(x): one Newton step on the reciprocal root (an ulp off) costs
    // nothing here and leaves no more rounding than a root and a division,
    // which took 143 instead of 140 us of a 256^3 stage
    const double y = rsqrt(x), S0 = f0 * y;
    double S = fma(0.5 * S0, fma(-(x * y), y, 1.0), S0);
    if (S0 != S0) S = 1.0;
    return (float)(S - S * dn);
}

// Position of the n-th (from 0) set bit of m, for n < popc(m): a binary
// search on the set-bit counts of halves, quarters, ... (always 0..31).
__device__ __forceinline__ int nth_set_bit(unsigned m, int n) {
    int pos = 0;
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
        const unsigned low = m & ((1u << w) - 1u);
        const int c = __popc(low);
        if (n >= c) {
            n -= c;
            m >>= w;
            pos += w;
        } else {
            m = low;
        }
    }
    return pos;
}

// 3-input minimum / maximum (one instruction on sm_100)
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// One tile configuration: TX x TY cells per CTA (TX/2 threads per row
// group, RY rows per thread), RING plane slots in shared memory, MINB CTAs
// per SM the registers are limited for.
template <int TX_, int TY_, int RY_, int RING_, int MINB_>
struct TileCfg {
    static constexpr int TX = TX_, TY = TY_, RY = RY_, RING = RING_, MINB = MINB_;
    static constexpr int TPR = TX / 2;           // threads per row group
    static constexpr int NT = TPR * (TY / RY);   // threads per CTA
    static constexpr int NW = NT / 32;
    static constexpr int BX = TX + 8, BY = TY + 6;
    static constexpr int SLOT = (BX * BY + 31) / 32 * 32;  // floats per slot (128-byte aligned)
    static constexpr unsigned BOX_BYTES = BX * BY * 4;
    static_assert(NT % 32 == 0 && TY % RY == 0, "whole warps, whole row groups");
    static_assert(RING >= 8, "the ring holds the 7-plane stencil and one plane in flight");
    static_assert(BX <= 256 && BY <= 256 && (BX * 4) % 16 == 0, "TMA box limits");
    static constexpr size_t smem() { return (size_t)RING * SLOT * 4 + RING * sizeof(uint64_t) + (RING + 2) * sizeof(int); }
};

// The configurations the library is built with (id = position).
#define R3D_TILE_CFGS(X)        \
    X(0, 64, 8, 1, 16, 3)       \
    X(1, 64, 8, 2, 12, 4)       \
    X(2, 64, 16, 2, 10, 2)      \
    X(3, 32, 16, 2, 12, 4)      \
    X(4, 128, 8, 2, 8, 2)       \
    X(5, 64, 8, 1, 10, 4)       \
    X(6, 32, 16, 2, 12, 5)

#define R3D_CFG_TYPE(id, tx, ty, ry, ring, minb) using Cfg##id = TileCfg<tx, ty, ry, ring, minb>;
R3D_TILE_CFGS(R3D_CFG_TYPE)
#undef R3D_CFG_TYPE

// One work item: the TX x TY column (bx, by) over planes [bz*kc, bz*kc+kc)
// of one instance.  When a bounded wait gives up, the error flag is raised
// and the copies in flight are waited for.  The item's volume partials (when
// `volume`) go to partial_out[0..1].
// ISO: the three axes have bitwise-equal spacing constants (cubic cells), so
// axis 0's are used for all three and held once.
//
// Shared memory is a ring of RING plane boxes: the x and y stencils of
// plane k come from its box, the z stencil from the thread's own column in
// the seven boxes k-3..k+3.  Each box has a "full" mbarrier (the TMA copy
// landed).  After plane k the box of plane k-3 is refilled with plane
// k-3+RING by the last warp to count itself out of the box (a per-box
// release counter), so that warps drift apart where their work differs
// (interface-band cells in FP64, wall ghosts) instead of meeting at a CTA
// barrier every plane.
template <class C, bool REINI, int STAGE, bool ISO>
__device__ __forceinline__ void tile_item(const CUtensorMap* tmap, const TileArgs& a, int bx, int by, int bz,
                                          bool volume, unsigned char* smem_raw, double* red_a, double* red_b,
                                          double* partial_out) {
    constexpr int RY = C::RY, BX = C::BX, RING = C::RING, SLOT = C::SLOT;
    float* ring = reinterpret_cast<float*>(smem_raw);
    uint64_t* bar = reinterpret_cast<uint64_t*>(ring + RING * SLOT);  // full
    int* rel = reinterpret_cast<int*>(bar + RING);                    // release counters
    volatile int* s_abort = rel + RING;
    int* s_issued = rel + RING + 1;  // last plane issued

    const Layout& L = a.L;
    const int sy = (int)L.sy, sz = (int)L.sz;
    const int tid = threadIdx.x, lane = tid & 31;
    const int tx = tid % C::TPR, tg = tid / C::TPR;
    const int i0 = bx * C::TX + 2 * tx;
    const int jb = by * C::TY + tg * RY;  // the thread's first row
    const int k0 = bz * a.kc;
    const int k1 = min(k0 + a.kc, L.nz);
    const int xbox = bx * C::TX + L.gx - 4;  // 16-byte aligned x start
    const int ybox = by * C::TY + L.gy - 3;
    const int pfirst = k0 - 3;  // first plane staged (ring position 0)
    const int plast = k1 + 2;   // last plane staged
    const int own = (tg * RY + 3) * BX + 2 * tx + 4;  // the thread's first two cells in a box
    // The thread's cells within a plane, as unsigned offsets from the plane's
    // (CTA-uniform) base pointers, so a load or store costs no 64-bit address
    // arithmetic per thread.  Loads are unconditional: a thread outside the
    // grid reads the nearest cell pair of its rows instead (the pair after
    // the last cell ends in the ghost layer), and its values go nowhere.
    const unsigned col0 = (unsigned)((jb + L.gy) * sy + (i0 + L.gx));
    unsigned ld[RY];
    // bits per row r (shifted by 8 r): 1 first cell inside, 2 second cell
    // inside, 4 x-min wall, 8 x-max wall (second cell), 16 x-max wall (first
    // cell), 32 y-min wall, 64 y-max wall
    unsigned flags = 0;
#pragma unroll
    for (int r = 0; r < RY; ++r) {
        const int j = jb + r;
        ld[r] = (unsigned)((min(j, L.ny - 1) + L.gy) * sy + (min(i0, (L.nx - 1) & ~1) + L.gx));
        const bool in0 = i0 < L.nx && j < L.ny, in1 = i0 + 1 < L.nx && j < L.ny;
        const unsigned f = (in0 ? 1u : 0u) | (in1 ? 2u : 0u) | (in0 && i0 == 0 ? 4u : 0u) |
                           (in1 && i0 + 1 == L.nx - 1 ? 8u : 0u) | (in0 && !in1 ? 16u : 0u) |
                           (in0 && j == 0 ? 32u : 0u) | (in0 && j == L.ny - 1 ? 64u : 0u);
        flags |= f << (8 * r);
    }
    const unsigned ldm = (unsigned)((min(jb, L.ny - 1) + L.gy - 1) * sy + (min(i0, (L.nx - 1) & ~1) + L.gx));

    if (tid == 0) {
        for (int s = 0; s < RING; ++s) {
            mbar_init(bar + s, 1);
            rel[s] = 0;
        }
        *s_abort = 0;
        mbar_fence_init();
        for (int p = pfirst; p <= min(pfirst + RING - 1, plast); ++p) {
            const int s = p - pfirst;
            mbar_expect_tx(bar + s, C::BOX_BYTES);
            tma_load_3d(ring + s * SLOT, tmap, bar + s, xbox, ybox, p + L.gz);
            *s_issued = p;
        }
    }
    __syncthreads();

    // planes k0-3 .. k0+2: the first window without its top plane
    const long long spin = a.spin > 0 ? a.spin : kSpin;
    bool ok = true;
#pragma unroll
    for (int m = 0; m < 6; ++m) ok = ok && mbar_wait_bounded(bar + m, 0, spin);
    // timeout-path test: the second completion of box 0 needs a refill that
    // only the plane loop issues, so this wait gives up after `spin` tries
    if (a.wait_test) ok = ok && mbar_wait_bounded(bar, 1, spin);

    const float vs = (float)*a.vscale;
    const float dtc = REINI ? a.dtr : (float)*a.dt;
    // plane base pointers, advanced with k
    const size_t c0 = (size_t)(k0 + L.gz) * (size_t)L.sz;
    const float *pu = a.u + c0, *pv = a.v + c0, *pw = a.w + c0, *pf = a.fn + c0;
    float* po = a.out + c0;
    float2 wprev[RY];
#pragma unroll
    for (int r = 0; r < RY; ++r)
        if (!REINI) wprev[r] = __ldg(reinterpret_cast<const float2*>(pw - sz + ld[r]));
    double vol_a = 0.0, vol_b = 0.0;

    // cell-local global operands of a plane (velocities, step start value),
    // fetched one plane ahead so their latency overlaps the current plane;
    // v on the face below row r is v of row r-1 for r > 0
    float2 nu[RY], nv[RY], nw[RY], nfn[RY], nvm0;
    float num[RY];
    auto fetch = [&]() {
#pragma unroll
        for (int r = 0; r < RY; ++r) {
            if (!REINI) {
                nu[r] = __ldg(reinterpret_cast<const float2*>(pu + ld[r]));
                num[r] = __ldg(pu + ld[r] - 1);
                nv[r] = __ldg(reinterpret_cast<const float2*>(pv + ld[r]));
                nw[r] = __ldg(reinterpret_cast<const float2*>(pw + ld[r]));
            }
            // the step start value may be this stage's output (stage 3): plain
            // loads, and of the thread's own cells alone
            if (STAGE == 2 || (STAGE == 3 && ((flags >> (8 * r)) & 1u))) nfn[r] = *reinterpret_cast<const float2*>(pf + ld[r]);
        }
        if (!REINI) nvm0 = __ldg(reinterpret_cast<const float2*>(pv + ldm));
        pu += sz;
        pv += sz;
        pw += sz;
        pf += sz;
    };
    fetch();

    constexpr int AY = ISO ? 0 : 1, AZ = ISO ? 0 : 2;
    int z[7];
#pragma unroll
    for (int m = 0; m < 6; ++m) z[m + 1] = m * SLOT + own;
    int sb = 0;          // ring slot of position n = k - k0 (plane k-3)
    int ws = 6, wp = 0;  // ring slot and phase parity of position n + 6 (plane k+3)
    for (int k = k0; k < k1; ++k, po += sz) {
        ok = __all_sync(0xffffffffu, ok && mbar_wait_bounded(bar + ws, (uint32_t)wp, spin));
        // a warp whose wait gave up leaves; the boxes it no longer releases
        // are not refilled, so the other warps' waits give up in turn
        if (!ok) {
            *s_abort = 1;
            break;
        }
        // the thread's own column in the boxes of planes k-3 .. k+3 (ring
        // offsets), moved on by one plane
#pragma unroll
        for (int m = 0; m < 6; ++m) z[m] = z[m + 1];
        z[6] = ws * SLOT + own;
        const float* zc[7];
#pragma unroll
        for (int m = 0; m < 7; ++m) zc[m] = ring + z[m];
        const float* sl = zc[3];

        // y stencil values of all RY rows, first and second differences
        float2 DY[RY + 5], EY[RY + 4], MY[RY];
        float2 fy2[RY], fy4[RY];
        {
            float2 fy[RY + 6];
#pragma unroll
            for (int m = 0; m < RY + 6; ++m) fy[m] = *reinterpret_cast<const float2*>(sl + (m - 3) * BX);
#pragma unroll
            for (int m = 0; m < RY + 5; ++m) DY[m] = sub2(fy[m + 1], fy[m]);
#pragma unroll
            for (int m = 0; m < RY + 4; ++m) EY[m] = sub2(DY[m + 1], DY[m]);
#pragma unroll
            for (int r = 0; r < RY; ++r) { fy2[r] = fy[r + 2]; fy4[r] = fy[r + 4]; MY[r] = sub2(fy4[r], fy2[r]); }
        }
        // this plane's operands, then the next plane's loads in flight
        // through the whole computation of this one
        float2 fnr[RY], ucr[RY], vcr[RY], wcr[RY], vm0;
        float umr[RY];
#pragma unroll
        for (int r = 0; r < RY; ++r) {
            if (STAGE != 1) fnr[r] = nfn[r];
            if (!REINI) { ucr[r] = nu[r]; vcr[r] = nv[r]; wcr[r] = nw[r]; umr[r] = num[r]; }
        }
        if (!REINI) vm0 = nvm0;
        if (k + 1 < k1) fetch();

        float2 f0[RY], Lc[RY];
        bool bandx[RY], bandy[RY];
#pragma unroll
        for (int r = 0; r < RY; ++r) {
            // x stencil: the row's columns 2tx .. 2tx+9 (the cells at 2tx+4, 2tx+5)
            float xv[10], dx[9], ex[8];
            {
                const float* rp = sl + r * BX - 4;
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    const float2 t = *reinterpret_cast<const float2*>(rp + 2 * q);
                    xv[2 * q] = t.x;
                    xv[2 * q + 1] = t.y;
                }
            }
#pragma unroll
            for (int m = 1; m < 8; ++m) dx[m] = xv[m + 1] - xv[m];
#pragma unroll
            for (int m = 2; m < 8; ++m) ex[m] = dx[m] - dx[m - 1];  // about column m
            float2 DZ[6], EZ[5], fz2, fz4;
            {
                float2 fz[7];
#pragma unroll
                for (int m = 0; m < 7; ++m) fz[m] = *reinterpret_cast<const float2*>(zc[m] + r * BX);
#pragma unroll
                for (int m = 0; m < 6; ++m) DZ[m] = sub2(fz[m + 1], fz[m]);
#pragma unroll
                for (int m = 0; m < 5; ++m) EZ[m] = sub2(DZ[m + 1], DZ[m]);
                fz2 = fz[2];
                fz4 = fz[4];
            }
            f0[r] = make_float2(xv[4], xv[5]);
            const float2 mx = make_float2(xv[5] - xv[3], xv[6] - xv[4]), mz = sub2(fz4, fz2);
            const float2 EX[5] = {make_float2(ex[2], ex[3]), make_float2(ex[3], ex[4]), make_float2(ex[4], ex[5]),
                                  make_float2(ex[5], ex[6]), make_float2(ex[6], ex[7])};
            bandx[r] = bandy[r] = false;
            if (!REINI) {
                // the derivatives come out as 2 h times themselves
                const float2 vm = r == 0 ? vm0 : vcr[r - 1];
                const float qv = 0.25f * vs;
                const float2 ia = mul2(f2(qv * a.rh[0]), add2(make_float2(umr[r], ucr[r].x), ucr[r]));
                const float2 ja = mul2(f2(qv * a.rh[AY]), add2(vcr[r], vm));
                const float2 ka = mul2(f2(qv * a.rh[AZ]), add2(wcr[r], wprev[r]));
                wprev[r] = wcr[r];
                const float2 gx = deriv2(EX, mx, ia.x < 0.f, ia.y < 0.f, a.psi1[0], a.psi2[0]);
                const float2 gy = deriv2(EY + r, MY[r], ja.x < 0.f,
                                         ja.y < 0.f, a.psi1[AY], a.psi2[AY]);
                const float2 gz = deriv2(EZ, mz, ka.x < 0.f, ka.y < 0.f, a.psi1[AZ],
                                         a.psi2[AZ]);
                Lc[r] = fma2(ka, gz, fma2(ja, gy, mul2(ia, gx)));  // -L
            } else {
                // Godunov selection per axis (src/reinidisc_f.cpp:70-109) on the
                // backward and forward differences m, p, with s the sign of
                // the cell:
                //   minus side: s m > 0 and s (m + p) > 0,
                //   plus side:  s p < 0 and s (m + p) < 0, else 0.
                // m + p is the central difference M: the plus side where
                // s M < 0, and the side's own difference has to have M's sign.
                const float2 fc = f0[r];
                const float2 sg = make_float2(fc.x > -1.0e-8f ? 1.f : -1.f, fc.y > -1.0e-8f ? 1.f : -1.f);
                float2 g2 = make_float2(0.f, 0.f);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const float2 dm = d == 0 ? make_float2(dx[3], dx[4]) : d == 1 ? DY[r + 2] : DZ[2];
                    const float2 dp = d == 0 ? make_float2(dx[4], dx[5]) : d == 1 ? DY[r + 3] : DZ[3];
                    const float2 M = d == 0 ? mx : d == 1 ? MY[r] : mz;
                    const float2 sM = mul2(M, sg);
                    const bool px = sM.x < 0.f, py = sM.y < 0.f;
                    const float2 side = mul2(sel2(px, py, dp, dm), M);
                    const int ad = ISO ? 0 : d;
                    float2 g = deriv2(d == 0 ? EX : d == 1 ? EY + r : EZ, M, px, py, a.psi1[ad], a.psi2[ad]);
                    if (!ISO) g = mul2(f2(a.rh[d]), g);
                    g.x = side.x > 0.f ? g.x : 0.f;
                    g.y = side.y > 0.f ? g.y : 0.f;
                    g2 = fma2(g, g, g2);
                }
                // the derivatives came out doubled (ISO: and times h)
                const float sc = ISO ? 0.25f * a.rh[0] * a.rh[0] : 0.25f;
                g2 = mul2(f2(sc), g2);
                const float2 dn = make_float2(sqrt_approx(g2.x), sqrt_approx(g2.y));
                const float2 dl = f2(a.deltax);
                const float2 den = fma2(mul2(mul2(dn, dn), dl), dl, mul2(fc, fc));
                float2 S = mul2(fc, make_float2(rsqrtf(den.x), rsqrtf(den.y)));
                if (S.x != S.x) S.x = 1.f;
                if (S.y != S.y) S.y = 1.f;
                Lc[r] = sub2(mul2(S, dn), S);  // -L = S |grad| - S
                // interface band: the 7-point stencil changes sign, i.e. neither
                // all values >= 0 (min >= 0) nor all < 0 (max < 0)
                const float lox = min3f(min3f(fc.x, xv[3], xv[5]), min3f(fy2[r].x, fy4[r].x, fz2.x), fz4.x);
                const float hix = max3f(max3f(fc.x, xv[3], xv[5]), max3f(fy2[r].x, fy4[r].x, fz2.x), fz4.x);
                const float loy = min3f(min3f(fc.y, xv[4], xv[6]), min3f(fy2[r].y, fy4[r].y, fz2.y), fz4.y);
                const float hiy = max3f(max3f(fc.y, xv[4], xv[6]), max3f(fy2[r].y, fy4[r].y, fz2.y), fz4.y);
                bandx[r] = lox < 0.f && hix >= 0.f;
                bandy[r] = loy < 0.f && hiy >= 0.f;
            }
        }
        bool band_here = false;
#pragma unroll
        for (int r = 0; r < RY; ++r) band_here = band_here || bandx[r] || bandy[r];
        // one vote for the plane: most warps hold no band cell in it
        if (REINI && __any_sync(0xffffffffu, band_here)) {
            if (a.f49 == 0) {
#pragma unroll
                for (int r = 0; r < RY; ++r) {
                    if (bandx[r]) Lc[r].x = 0.f;  // src/reinidisc_fsf.cpp:70-72
                    if (bandy[r]) Lc[r].y = 0.f;
                }
            } else if (a.band64) {
                // The band cells of the warp's RY rows are dealt out to its
                // lanes, stencils from shared memory, results back to the owning
                // lanes by shuffles.  A round takes ten cells with one axis per
                // lane, or (more than twenty left) 32 cells with all three: an
                // FP64 WENO evaluation is a chain of ~600 cycles, so a curved
                // interface, which leaves a few cells per row, is served in one
                // such latency instead of three.
                unsigned mk[2 * RY];
                int end[2 * RY];  // cells of the masks up to and including this one
                int total = 0;
#pragma unroll
                for (int q = 0; q < 2 * RY; ++q) {
                    mk[q] = __ballot_sync(0xffffffffu, q & 1 ? (flags >> (8 * (q >> 1)) & 2u) && bandy[q >> 1]
                                                          : (flags >> (8 * (q >> 1)) & 1u) && bandx[q >> 1]);
                    total += __popc(mk[q]);
                    end[q] = total;
                }
                const unsigned below = (1u << lane) - 1u;
                for (int base = 0; base < total;) {
                    const bool wide = total - base > 20;
                    const int cells = wide ? 32 : 10;
                    const int b = base + (wide ? lane : lane / 3);
                    double g2 = 0.0;
                    float fcen = 0.f, res = 0.f;
                    if (b < total && (wide || lane < 30)) {
                        int q = 0;
#pragma unroll
                        for (int m = 0; m + 1 < 2 * RY; ++m) q += b >= end[m];
                        unsigned mq = mk[0];
                        int first = 0;
#pragma unroll
                        for (int m = 1; m < 2 * RY; ++m)
                            if (q == m) {
                                mq = mk[m];
                                first = end[m - 1];
                            }
                        const int st = (tid & ~31) + nth_set_bit(mq, b - first);  // the thread that owns the cell
                        const int oc = ((st / C::TPR) * RY + (q >> 1) + 3) * BX + 2 * (st % C::TPR) + 4 + (q & 1);
                        const float* cen = sl - own + oc;
                        fcen = *cen;
                        const int ax0 = wide ? 0 : lane - 3 * (lane / 3), ax1 = wide ? 3 : ax0 + 1;
                        for (int ax = ax0; ax < ax1; ++ax) {
                            float f[7];
#pragma unroll
                            for (int m = 0; m < 7; ++m) {
                                const float* pz = zc[m] - own + oc;
                                f[m] = ax == 2 ? *pz : cen[(m - 3) * (ax == 0 ? 1 : BX)];
                            }
                            g2 += band_axis(f[0], f[1], f[2], f[3], f[4], f[5], f[6], ax == 0 ? a.rh[0] : ax == 1 ? a.rh[1] : a.rh[2],
                                            ax == 0 ? a.beps[0] : ax == 1 ? a.beps[1] : a.beps[2]);
                        }
                    }
                    if (!wide) {
                        const double gy = __shfl_down_sync(0xffffffffu, g2, 1), gz = __shfl_down_sync(0xffffffffu, g2, 2);
                        g2 = (g2 + gy) + gz;
                    }
                    if (b < total) res = -band_rhs(fcen, g2, a.deltax);
#pragma unroll
                    for (int q = 0; q < 2 * RY; ++q) {
                        const int mine = (q ? end[q - 1] : 0) + __popc(mk[q] & below) - base;
                        const float v = __shfl_sync(0xffffffffu, res, (wide ? mine : 3 * mine) & 31);
                        if (((mk[q] >> lane) & 1u) && mine >= 0 && mine < cells) {
                            if (q & 1) Lc[q >> 1].y = v;
                            else Lc[q >> 1].x = v;
                        }
                    }
                    base += cells;
                }
            }
        }

        // the warp's shared-memory reads of this plane are done, so it counts
        // itself out of the box of plane k-3 (before its global stores and
        // loads, so the fence waits on nothing in flight), and the last warp
        // out refills the box with plane k-3+RING
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            if (atomicAdd(rel + sb, 1) == C::NW - 1) {
                __threadfence_block();
                rel[sb] = 0;
                if (k - 3 + RING <= plast) {
                    fence_proxy_async();
                    mbar_expect_tx(bar + sb, C::BOX_BYTES);
                    tma_load_3d(ring + sb * SLOT, tmap, bar + sb, xbox, ybox, k - 3 + RING + L.gz);
                    atomicMax(s_issued, k - 3 + RING);
                }
            }
        }

#pragma unroll
        for (int r = 0; r < RY; ++r) {
            // RK combine (src/levelset_RK3.cpp:121-156, src/reini_RK3.cpp:118-135)
            float2 val;
            const float2 sdl = fma2(f2(-dtc), Lc[r], f0[r]);  // stage input + dt L
            if (STAGE == 1) {
                val = sdl;
            } else {
                if (STAGE == 2) val = fma2(f2(0.75f), fnr[r], mul2(f2(0.25f), sdl));
                else val = fma2(f2(1.0f / 3.0f), fnr[r], mul2(f2(2.0f / 3.0f), sdl));
            }
            const unsigned fl = flags >> (8 * r);
            float* o = po + (col0 + (unsigned)(r * sy));
            if (fl & 2u) *reinterpret_cast<float2*>(o) = val;
            else if (fl & 1u) *o = val.x;
            // wall ghost copies (src/gc_neumann.cpp:29-54)
            if (fl & 0x1cu) {
                // x-min: three ghosts and the padding slot before them, 16-byte aligned
                if (fl & 4u) *reinterpret_cast<float4*>(o - 4) = make_float4(val.x, val.x, val.x, val.x);
                if (fl & 8u) {
                    *reinterpret_cast<float2*>(o + 2) = make_float2(val.y, val.y);
                    o[4] = val.y;
                }
                if (fl & 16u) { o[1] = val.x; o[2] = val.x; o[3] = val.x; }
            }
            if (fl & 0x60u) {
                // ny >= 2 here (ny = 1 is a 2D grid), so never both y walls
                const int dir = fl & 32u ? -sy : sy;
#pragma unroll
                for (int q = 1; q <= 3; ++q) {
                    o[q * dir] = val.x;
                    if (fl & 2u) o[q * dir + 1] = val.y;
                }
            }
            if (k == 0 || k == L.nz - 1) {
                // a slab face's ghosts come from the neighbour
                if (k == 0 && !(L.io & kHaloZLo) && (fl & 1u))
                    for (int q = 1; q <= 3; ++q) {
                        o[-(long long)q * sz] = val.x;
                        if (fl & 2u) o[-(long long)q * sz + 1] = val.y;
                    }
                if (k == L.nz - 1 && !(L.io & kHaloZHi) && (fl & 1u))
                    for (int q = 1; q <= 3; ++q) {
                        o[(long long)q * sz] = val.x;
                        if (fl & 2u) o[(long long)q * sz + 1] = val.y;
                    }
            }
            f0[r] = val;  // for the volume
        }
        if (volume) {
            // Smoothed Heaviside in FP64 (src/fluid_update_fsf.cpp:50-71).  The
            // cells inside the interface thickness, a few of a warp's 64 RY,
            // are dealt out to its lanes: one FP64 sine (and two divisions)
            // in all lanes at once instead of one per row and side with most
            // lanes idle: 17 us of a 256^3 step.
            const double PI_REF = 3.14159265359;
            unsigned mk[2 * RY];
            int end[2 * RY], total = 0;
#pragma unroll
            for (int q = 0; q < 2 * RY; ++q) {
                const double ph = q & 1 ? f0[q >> 1].y : f0[q >> 1].x;
                const bool in = (flags >> (8 * (q >> 1))) & (q & 1 ? 2u : 1u);
                const bool band = in && fabs(ph) <= a.psi;
                if (in && !band) {
                    if (ph > a.psi) vol_a += a.cellvol;
                    else vol_b += a.cellvol;
                }
                mk[q] = __ballot_sync(0xffffffffu, band);
                total += __popc(mk[q]);
                end[q] = total;
            }
            for (int base = 0; base < total; base += 32) {
                const int b = base + lane;
                int q = 0, before = 0;
                unsigned mq = mk[0];
#pragma unroll
                for (int m = 1; m < 2 * RY; ++m)
                    if (b >= end[m - 1]) {
                        q = m;
                        mq = mk[m];
                        before = end[m - 1];
                    }
                const int src = b < total ? nth_set_bit(mq, b - before) : 0;
                float v = 0.f;
#pragma unroll
                for (int m = 0; m < 2 * RY; ++m) {
                    const float c = __shfl_sync(0xffffffffu, m & 1 ? f0[m >> 1].y : f0[m >> 1].x, src);
                    if (q == m) v = c;
                }
                if (b < total) {
                    const double ph = v;
                    const double H = 0.5 * (1.0 + ph / a.psi + (1.0 / PI_REF) * sin((PI_REF * ph) / a.psi));
                    vol_a += a.cellvol * H;
                    vol_b += a.cellvol * (1.0 - H);
                }
            }
        }

        sb = sb + 1 == RING ? 0 : sb + 1;
        if (++ws == RING) {
            ws = 0;
            wp ^= 1;
        }
    }
    __syncthreads();
    const bool aborted = *s_abort != 0;

    if (aborted) {
        if (tid == 0) {
            atomicExch(a.err, 1);
            // wait (bounded) for every copy still in flight before leaving
            for (int p = pfirst; p <= *s_issued; ++p) {
                const int q = p - pfirst;
                mbar_wait_bounded(bar + (q % RING), (uint32_t)((q / RING) & 1));
            }
        }
        return;
    }
    if (volume) {
        for (int o = 16; o > 0; o >>= 1) {
            vol_a += __shfl_down_sync(0xffffffffu, vol_a, o);
            vol_b += __shfl_down_sync(0xffffffffu, vol_b, o);
        }
        if (lane == 0) { red_a[tid >> 5] = vol_a; red_b[tid >> 5] = vol_b; }
        __syncthreads();
        if (tid == 0) {
            double sa = 0.0, sb2 = 0.0;
            for (int q = 0; q < C::NW; ++q) { sa += red_a[q]; sb2 += red_b[q]; }
            partial_out[0] = sa;
            partial_out[1] = sb2;
        }
    }
}

template <class C, bool REINI, int STAGE, bool VOLUME, bool ISO>
__global__ void __launch_bounds__(C::NT, C::MINB) tile_kernel(const __grid_constant__ CUtensorMap tmap,
                                                              const __grid_constant__ TileArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ double red_a[C::NW], red_b[C::NW];
    const long long b = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    tile_item<C, REINI, STAGE, ISO>(&tmap, a, blockIdx.x, blockIdx.y, blockIdx.z, VOLUME, smem_raw, red_a, red_b,
                               a.partial + 2 * b);
}

// Batched form: CTA t takes item t of the tiled members (member m owns items
// [tile0[m], tile0[m+1]); item = (bx, by, bz) of that member), so the
// hardware hands a CTA that is done its SM's next item, whatever the items'
// work (FP64 interface band, wall ghosts); items taken by persistent CTAs
// from a counter paid a counter round trip, the retirement of the barriers
// and three CTA barriers each: 16 members of 64..160 cells an edge 1.64 ->
// 1.50 ms per step.  Reinitialisation pseudo-step q is skipped by members with
// f44 <= q; the last stage of a member's step adds its volume partials.
template <class C, bool REINI, int STAGE, bool ISO>
__global__ void __launch_bounds__(C::NT, C::MINB) batch_tile_kernel(const TiledMember* __restrict__ members,
                                                                    const CUtensorMap* __restrict__ maps,
                                                                    const long long* __restrict__ tile0, int nm,
                                                                    int q, double* __restrict__ vol_part) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ double red_a[C::NW], red_b[C::NW];
    __shared__ TileArgs sa;
    __shared__ int s_member;
    const long long t = blockIdx.x;
    if (threadIdx.x < 32) {
        // the last member whose first item is not after t
        const int lane = threadIdx.x;
        int m = -1;
        for (int base = 0; base < nm; base += 32) {
            const int n = __popc(__ballot_sync(0xffffffffu, base + lane < nm && __ldg(tile0 + base + lane) <= t));
            m = n ? base + n - 1 : m;
            if (n < 32) break;
        }
        static_assert(sizeof(TileArgs) % sizeof(int) == 0, "copied word by word");
        const int* src = reinterpret_cast<const int*>(&members[m].args);
        for (int e = lane; e < (int)(sizeof(TileArgs) / sizeof(int)); e += 32) reinterpret_cast<int*>(&sa)[e] = __ldg(src + e);
        __syncwarp();
        if (lane == 0) {
            s_member = m;
            sa.out = STAGE == 1 ? members[m].a1 : STAGE == 2 ? members[m].a2 : members[m].phi;
        }
    }
    __syncthreads();
    const int m = s_member;
    const int f44 = members[m].f44;
    if (REINI && f44 <= q) return;
    const bool volume = STAGE == 3 && (REINI ? q == f44 - 1 : f44 == 0);
    const long long lt = t - tile0[m];
    const int ntx = (sa.L.nx + C::TX - 1) / C::TX, nty = (sa.L.ny + C::TY - 1) / C::TY;
    const int bx = (int)(lt % ntx);
    const int by = (int)((lt / ntx) % nty);
    const int bz = (int)(lt / ((long long)ntx * nty));
    // the item's arguments in a thread-local copy: the plane loop reads them
    // across barriers, after which shared memory would be reread
    const TileArgs a = sa;
    tile_item<C, REINI, STAGE, ISO>(maps + 3 * m + (STAGE - 1), a, bx, by, bz, volume, smem_raw, red_a, red_b,
                                    vol_part + 2 * t);
}

// Face maxima over the cells of one item (x faces 0..nx-2, y 0..ny-2, z
// 0..nz-2, src/ietimestep.cpp:72-88) for every tiled member's item.
template <class C>
__global__ void __launch_bounds__(C::NT) batch_tile_vmax_kernel(const TiledMember* __restrict__ members,
                                                                const long long* __restrict__ tile0, int nm,
                                                                double* __restrict__ vmax_part) {
    __shared__ unsigned s[3][C::NW];
    const long long nt = tile0[nm];
    for (long long t = blockIdx.x; t < nt; t += gridDim.x) {
        int lo = 0, hi = nm - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (tile0[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
        const TileArgs& a = members[lo].args;
        const Layout& L = a.L;
        const long long lt = t - tile0[lo];
        const int ntx = (L.nx + C::TX - 1) / C::TX, nty = (L.ny + C::TY - 1) / C::TY;
        const int bx = (int)(lt % ntx), by = (int)((lt / ntx) % nty), bz = (int)(lt / ((long long)ntx * nty));
        const int tx = threadIdx.x % C::TPR, tg = threadIdx.x / C::TPR;
        const int i0 = bx * C::TX + 2 * tx;
        const int k0 = bz * a.kc, k1 = min(k0 + a.kc, L.nz);
        // |x| compared as the float's bit pattern with the sign cleared (exact)
        unsigned mu = 0u, mv = 0u, mw = 0u;
        for (int r = 0; r < C::RY; ++r) {
            const int j = by * C::TY + tg * C::RY + r;
            if (j >= L.ny || i0 >= L.nx) continue;
            const bool two = i0 + 1 < L.nx;
            const long long col = (long long)(j + L.gy) * L.sy + (i0 + L.gx);
            for (int k = k0; k < k1; ++k) {
                const long long c = (long long)(k + L.gz) * L.sz + col;
                float2 fu, fv, fw;
                if (two) {
                    fu = __ldg(reinterpret_cast<const float2*>(a.u + c));
                    fv = __ldg(reinterpret_cast<const float2*>(a.v + c));
                    fw = __ldg(reinterpret_cast<const float2*>(a.w + c));
                } else {
                    fu = make_float2(__ldg(a.u + c), 0.f);
                    fv = make_float2(__ldg(a.v + c), 0.f);
                    fw = make_float2(__ldg(a.w + c), 0.f);
                }
                if (i0 < L.nx - 1) mu = max(mu, __float_as_uint(fu.x) & 0x7fffffffu);
                if (i0 + 1 < L.nx - 1) mu = max(mu, __float_as_uint(fu.y) & 0x7fffffffu);
                if (j < L.ny - 1) mv = max(mv, max(__float_as_uint(fv.x) & 0x7fffffffu, __float_as_uint(fv.y) & 0x7fffffffu));
                if (k < L.nz - 1) mw = max(mw, max(__float_as_uint(fw.x) & 0x7fffffffu, __float_as_uint(fw.y) & 0x7fffffffu));
            }
        }
        mu = __reduce_max_sync(0xffffffffu, mu);
        mv = __reduce_max_sync(0xffffffffu, mv);
        mw = __reduce_max_sync(0xffffffffu, mw);
        const int w = threadIdx.x >> 5;
        if ((threadIdx.x & 31) == 0) { s[0][w] = mu; s[1][w] = mv; s[2][w] = mw; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int q = 1; q < C::NW; ++q) { mu = max(mu, s[0][q]); mv = max(mv, s[1][q]); mw = max(mw, s[2][q]); }
            vmax_part[3 * t] = (double)__uint_as_float(mu);
            vmax_part[3 * t + 1] = (double)__uint_as_float(mv);
            vmax_part[3 * t + 2] = (double)__uint_as_float(mw);
        }
        __syncthreads();
    }
}

// The ring needs more than the default 48 KB of dynamic shared memory, and a
// full shared-memory carveout lets several CTAs share an SM.
template <typename K>
bool tile_attr(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess &&
           cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100) == cudaSuccess;
}

template <class C, bool ISO>
bool cfg_prepare_iso(size_t b) {
    return tile_attr(tile_kernel<C, false, 1, false, ISO>, b) && tile_attr(tile_kernel<C, false, 2, false, ISO>, b) &&
           tile_attr(tile_kernel<C, false, 3, false, ISO>, b) && tile_attr(tile_kernel<C, false, 1, true, ISO>, b) &&
           tile_attr(tile_kernel<C, false, 2, true, ISO>, b) && tile_attr(tile_kernel<C, false, 3, true, ISO>, b) &&
           tile_attr(tile_kernel<C, true, 1, false, ISO>, b) && tile_attr(tile_kernel<C, true, 2, false, ISO>, b) &&
           tile_attr(tile_kernel<C, true, 3, false, ISO>, b) && tile_attr(tile_kernel<C, true, 1, true, ISO>, b) &&
           tile_attr(tile_kernel<C, true, 2, true, ISO>, b) && tile_attr(tile_kernel<C, true, 3, true, ISO>, b) &&
           tile_attr(batch_tile_kernel<C, false, 1, ISO>, b) && tile_attr(batch_tile_kernel<C, false, 2, ISO>, b) &&
           tile_attr(batch_tile_kernel<C, false, 3, ISO>, b) && tile_attr(batch_tile_kernel<C, true, 1, ISO>, b) &&
           tile_attr(batch_tile_kernel<C, true, 2, ISO>, b) && tile_attr(batch_tile_kernel<C, true, 3, ISO>, b);
}

template <class C>
bool cfg_prepare() {
    return cfg_prepare_iso<C, false>(C::smem()) && cfg_prepare_iso<C, true>(C::smem());
}

template <class C, bool ISO>
void launch_stage_cfg(const CUtensorMap& map, const TileArgs& a, bool reini, int stage, bool volume,
                      cudaStream_t st) {
    const dim3 grid((a.L.nx + C::TX - 1) / C::TX, (a.L.ny + C::TY - 1) / C::TY, (a.L.nz + a.kc - 1) / a.kc);
    const dim3 block(C::NT);
    const size_t sm = C::smem();
#define R3D_TL(R, S, V) tile_kernel<C, R, S, V, ISO><<<grid, block, sm, st>>>(map, a)
    if (reini) {
        if (stage == 1) { if (volume) R3D_TL(true, 1, true); else R3D_TL(true, 1, false); }
        else if (stage == 2) { if (volume) R3D_TL(true, 2, true); else R3D_TL(true, 2, false); }
        else { if (volume) R3D_TL(true, 3, true); else R3D_TL(true, 3, false); }
    } else {
        if (stage == 1) { if (volume) R3D_TL(false, 1, true); else R3D_TL(false, 1, false); }
        else if (stage == 2) { if (volume) R3D_TL(false, 2, true); else R3D_TL(false, 2, false); }
        else { if (volume) R3D_TL(false, 3, true); else R3D_TL(false, 3, false); }
    }
#undef R3D_TL
}

template <class C, bool ISO>
void launch_batch_cfg(const TiledMember* members, const CUtensorMap* maps, const long long* tile0, int nm,
                      bool reini, int stage, int q, double* vol_part, unsigned grid, cudaStream_t st) {
    const size_t sm = C::smem();
    const dim3 g(grid), block(C::NT);
#define R3D_BT(R, S) batch_tile_kernel<C, R, S, ISO><<<g, block, sm, st>>>(members, maps, tile0, nm, q, vol_part)
    if (reini) {
        if (stage == 1) R3D_BT(true, 1);
        else if (stage == 2) R3D_BT(true, 2);
        else R3D_BT(true, 3);
    } else {
        if (stage == 1) R3D_BT(false, 1);
        else if (stage == 2) R3D_BT(false, 2);
        else R3D_BT(false, 3);
    }
#undef R3D_BT
}

struct CfgInfo {
    int tx, ty, ry, ring, minb, threads;
    size_t smem;
};

const CfgInfo kCfgInfo[] = {
#define R3D_CFG_INFO(id, tx, ty, ry, ring, minb) {tx, ty, ry, ring, minb, Cfg##id::NT, Cfg##id::smem()},
    R3D_TILE_CFGS(R3D_CFG_INFO)
#undef R3D_CFG_INFO
};
constexpr int kNumCfg = sizeof(kCfgInfo) / sizeof(kCfgInfo[0]);

const CfgInfo& info(int cfg) { return kCfgInfo[(cfg >= 0 && cfg < kNumCfg) ? cfg : 0]; }

}  // namespace

int tile_cfg_count() { return kNumCfg; }

int tile_cfg_describe(int cfg, int* tx, int* ty, int* ry, int* ring, int* threads) {
    if (cfg < 0 || cfg >= kNumCfg) return 1;
    const CfgInfo& c = kCfgInfo[cfg];
    if (tx) *tx = c.tx;
    if (ty) *ty = c.ty;
    if (ry) *ry = c.ry;
    if (ring) *ring = c.ring;
    if (threads) *threads = c.threads;
    return 0;
}

int tile_ctas_per_sm(int cfg) { return info(cfg).minb; }

// Measured over every configuration and chunk on grids from 32^3 to
// 512 x 128 x 256 (us per stage, this choice / the best of the sweep /
// configuration 0 with 16 planes, the former default):
//   convection        64^3 7.4 / 6.7 / 20   128^3 21.3 / 20.6 / 26
//                     96^3 12.7 / 12.0 / 22  201x97x153 34 / 34 / 40  256^3 122 / 122 / 150
//   reinitialisation  64^3 10.3 / 8.8 / 45  128^3 27.7 / 27.2 / 50
//                     201x97x153 43 / 43 / 63  256^3 133 / 133 / 165
// Shape: the 64 x 8 tile for the convection (four CTAs per SM; it spills in
// the 96 registers of the fifth), 32 x 16 at five CTAs for the
// reinitialisation, or the other shape where it pads the grid less.  Chunk:
// a plane takes about 1 us alone on an SM and 2 us beside three others, an
// item 4 us on top, so the chunk shrinks until the items fill the device
// about twice over; the reinitialisation's items hold unequal numbers of FP64
// band cells and want three times as many.
void tile_default(const Layout& L, int sms, bool reini, int* cfg, int* kc) {
    auto columns = [&](int c) {
        return (long long)((L.nx + info(c).tx - 1) / info(c).tx) * ((L.ny + info(c).ty - 1) / info(c).ty);
    };
    auto padded = [&](int c) { return columns(c) * info(c).tx * info(c).ty; };
    const int first = reini ? 6 : 1, other = reini ? 1 : 3;
    *cfg = 100 * padded(other) < 97 * padded(first) ? other : first;
    const double waves = (double)(columns(*cfg) * L.nz) / ((double)sms * info(*cfg).minb);  // of one-plane items
    const int want = (int)(waves / (reini ? 7.0 : 2.2) + 0.5);
    const int lo = reini ? 1 : 2, hi = reini ? 8 : 10;
    *kc = want < lo ? lo : want > hi ? hi : want;
}

// Sets the attributes of every instantiation once per device.
bool tile_prepare() {
    static bool done[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    if (dev >= 0 && dev < 64 && done[dev]) return true;
    bool ok = true;
#define R3D_CFG_PREP(id, tx, ty, ry, ring, minb) ok = ok && cfg_prepare<Cfg##id>();
    R3D_TILE_CFGS(R3D_CFG_PREP)
#undef R3D_CFG_PREP
    if (!ok) {
        cudaGetLastError();
        return false;
    }
    if (dev >= 0 && dev < 64) done[dev] = true;
    return true;
}

long long tile_items_of(const Layout& L, int kc, int cfg) {
    const dim3 g = tile_grid(L, kc, cfg);
    return (long long)g.x * g.y * g.z;
}

int launch_batch_tile_stage(const TiledMember* members, const CUtensorMap* maps, const long long* tile0, int nm,
                            int cfg, bool iso, bool reini, int stage, int q, double* vol_part,
                            unsigned grid, cudaStream_t st) {
    tile_prepare();  // a failure here makes the launch below fail, which the caller reports
#define R3D_BATCH(C, I) launch_batch_cfg<C, I>(members, maps, tile0, nm, reini, stage, q, vol_part, grid, st)
    switch (cfg) {
#define R3D_CFG_CASE(id, tx, ty, ry, ring, minb) \
    case id: if (iso) R3D_BATCH(Cfg##id, true); else R3D_BATCH(Cfg##id, false); break;
        R3D_TILE_CFGS(R3D_CFG_CASE)
#undef R3D_CFG_CASE
        default: if (iso) R3D_BATCH(Cfg0, true); else R3D_BATCH(Cfg0, false);
    }
#undef R3D_BATCH
    return 1;
}

int launch_batch_tile_vmax(const TiledMember* members, const long long* tile0, int nm, int cfg, double* vmax_part,
                           unsigned grid, cudaStream_t st) {
    switch (cfg) {
#define R3D_CFG_CASE(id, tx, ty, ry, ring, minb) \
    case id: batch_tile_vmax_kernel<Cfg##id><<<grid, Cfg##id::NT, 0, st>>>(members, tile0, nm, vmax_part); break;
        R3D_TILE_CFGS(R3D_CFG_CASE)
#undef R3D_CFG_CASE
        default: batch_tile_vmax_kernel<Cfg0><<<grid, Cfg0::NT, 0, st>>>(members, tile0, nm, vmax_part);
    }
    return 1;
}

int encode_plane_map(const Layout& L, const float* base, int cfg, CUtensorMap* out, std::string* why) {
    using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn) {
            cudaGetLastError();
            if (why) *why = "cuTensorMapEncodeTiled unavailable";
            return 1;
        }
        encode = reinterpret_cast<EncodeFn>(fn);
    }
    // strides must be multiples of 16 bytes and the base 16-byte aligned
    if ((L.px * 4) % 16 != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0) {
        if (why) *why = "field not 16-byte aligned for TMA";
        return 1;
    }
    const CfgInfo& c = info(cfg);
    const cuuint64_t dims[3] = {(cuuint64_t)L.px, (cuuint64_t)L.py, (cuuint64_t)L.pz};
    const cuuint64_t strides[2] = {(cuuint64_t)L.px * 4, (cuuint64_t)L.px * L.py * 4};
    const cuuint32_t box[3] = {(cuuint32_t)(c.tx + 8), (cuuint32_t)(c.ty + 6), 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box,
                              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        if (why) *why = "cuTensorMapEncodeTiled failed";
        return 1;
    }
    return 0;
}

size_t tile_smem_bytes(int cfg) { return info(cfg).smem; }

dim3 tile_grid(const Layout& L, int kc, int cfg) {
    const CfgInfo& c = info(cfg);
    return dim3((L.nx + c.tx - 1) / c.tx, (L.ny + c.ty - 1) / c.ty, (L.nz + kc - 1) / kc);
}

int launch_tile_stage(const CUtensorMap& map, const TileArgs& a, int cfg, bool reini, int stage, bool volume,
                      cudaStream_t st) {
    tile_prepare();  // a failure here makes the launch below fail, which the caller reports
    const bool iso = tile_args_iso(a);
#define R3D_STAGE(C, I) launch_stage_cfg<C, I>(map, a, reini, stage, volume, st)
    switch (cfg) {
#define R3D_CFG_CASE(id, tx, ty, ry, ring, minb) \
    case id: if (iso) R3D_STAGE(Cfg##id, true); else R3D_STAGE(Cfg##id, false); break;
        R3D_TILE_CFGS(R3D_CFG_CASE)
#undef R3D_CFG_CASE
        default: if (iso) R3D_STAGE(Cfg0, true); else R3D_STAGE(Cfg0, false);
    }
#undef R3D_STAGE
    return 1;
}

}  // namespace r3d
