// 3-D mesh transforms of the Poisson solve, axis by axis, with the
// Fourier-space operators of pmwd/gravity.py:9-72 fused into the x axis.
//
// Forward force (rho -> three acceleration meshes):
//   k_rows_r2c   z axis:  real rows -> half rows
//   k_cols_fwd   y axis:  half rows -> H(x; ky, kz)
//   k_xaxis_fwd  x axis:  P = -(c / k^2) FFT_x(H),  G_0 = IFFT_x(-i kx P),
//                         Q = IFFT_x(P)
//   k_cols_inv   y axis:  IFFT_y of G_0, -i ky Q and -i kz Q (ky and kz are
//                         constant along x, so Q serves both)
//   k_rows_c2r   z axis:  half rows -> real rows
// Force VJP (cotangents of the three meshes -> cotangent of rho), the exact
// transpose:
//   k_rows_r2c; k_cols_adj (C_0 = FFT_y, D = i ky FFT_y(C_1) + i kz FFT_y(C_2));
//   k_xaxis_adj (S = IFFT_x(-(c / k^2) [i kx FFT_x(C_0) + FFT_x(D)]));
//   k_cols_inv; k_rows_c2r.
// Two spectra instead of three pass through the x axis in either direction.
// Square planes up to 128 x 128: k_plane_fwd and k_plane_inv do both axes of a plane
// (pmx_mesh_plane.cu).
//
// Every length-N transform is N = R1 * R2: radix-R1 DFTs of R2-strided
// elements in registers, twiddles, ONE exchange through shared memory,
// radix-R2 DFTs, straight from and to global memory -- no staging copies.
// At N = 1024 a block of 128 threads holds 4 columns (34 KB), so several
// blocks share an SM and one's loads overlap another's arithmetic.
//
// Measured at 1024^3 (GB300, ms): rows r2c 1.43, cols fwd 1.51, x fwd 3.88,
// cols inv 4.80, rows c2r 3 x 1.30; adjoint rows 4.28, cols 5.68, x 3.75, cols
// inv 1.68, rows 1.30.  The cuFFT plane transforms and the tiled x pass that
// they replace: r2c 3.4, x 6.8, c2r 11.1; adjoint 10.1, 8.5, 3.7.
//
// Layouts.  Strided axes make the memory system, not the arithmetic, the
// bound: at 1024^3 an x-axis column in a natural (x, ky, kz) array is read in
// 64-byte pieces 4.2 MB apart, 2.5 TB/s at best.  Two blocked layouts of
// complex64 in units of 32 values (256 bytes, one warp-wide access) avoid
// that; kz is padded to a multiple of 4:
//   half rows ("nat"):  (plane, y / 8, kz / 4, y % 8, kz % 4)
//   spectra ("spec"):   (x / 8, ky, kz / 4, x % 8, kz % 4)
// The z kernels write nat from 8 rows at a time and the x kernels touch spec
// in whole 256-byte blocks; only the y kernels see 32-byte pieces (on the
// spec side), and the blocks of eight x-planes that fill one 256-byte block
// run next to each other, so L2 merges them.

#pragma once

#include <cuda_runtime.h>

#include "pmx_dft.cuh"
#include "pmx_internal.cuh"

namespace pmx {

// N = R1 * R2, R1 >= R2 except 768; T columns per block.
template <int N>
struct Fac;
template <> struct Fac<64> { static constexpr int R1 = 8, R2 = 8; };
template <> struct Fac<96> { static constexpr int R1 = 12, R2 = 8; };
template <> struct Fac<128> { static constexpr int R1 = 16, R2 = 8; };
template <> struct Fac<192> { static constexpr int R1 = 24, R2 = 8; };
template <> struct Fac<256> { static constexpr int R1 = 16, R2 = 16; };
template <> struct Fac<384> { static constexpr int R1 = 24, R2 = 16; };
template <> struct Fac<512> { static constexpr int R1 = 32, R2 = 16; };
template <> struct Fac<768> { static constexpr int R1 = 24, R2 = 32; };
template <> struct Fac<1024> { static constexpr int R1 = 32, R2 = 32; };

// Block of T columns of length N: T * R2 threads, one radix-R1 DFT each in the
// first stage.
template <int N_, int T_>
struct TileCfg {
    static constexpr int N = N_, T = T_;
    static constexpr int R1 = Fac<N>::R1, R2 = Fac<N>::R2;
    static constexpr int TH = T * R2;
    // shared exchange buffer: element (k1, b) of column t at k1 * GS + b * T + t;
    // R2 + 1 odd keeps both sides free of bank conflicts
    static constexpr int GS = (R2 + 1) * T;
    static constexpr int BUF = R1 * GS;
};

// x axis: T consecutive kz of one ky (whole spec blocks of 4 kz).
template <int N>
using XCol = TileCfg<N, 128 / Fac<N>::R2 < 4 ? 4 : 128 / Fac<N>::R2>;

// y axis: XP = T / 4 consecutive x-planes times 4 kz, so that a block touches
// XP * 32 contiguous bytes of a spec block at a time.  Larger XP (256-thread
// blocks) makes wider pieces but lost to the 128-thread blocks' finer overlap of
// loads and arithmetic: 5.1 against 4.8 ms for the three inverse transforms at
// 1024^3, 0.55 against 0.50 at 512^3.
template <int N>
using YCol = XCol<N>;

// Half length L = R1 * R2 of a row transform.  R1 / 2 threads share a row:
// thread 0 holds the groups k1 = 0 and R1 / 2 of the radix-R2 side, thread i
// the groups i and R1 - i, so that every pair Z[k], Z[L - k] that the
// real-input split combines meets in one thread's registers.
template <int L>
struct RowCfg;
#define PMX_ROW_CFG(L_, R1_, R2_)                 \
    template <>                                   \
    struct RowCfg<L_> {                           \
        static constexpr int R1 = R1_, R2 = R2_;  \
        static constexpr int TPR = R1 / 2;        \
        static constexpr int ROWS = 128 / TPR;    \
        static constexpr int TH = 128;            \
        static constexpr int S = R2 + 1;          \
        /* rows 16, 8 or 4 values apart (mod 16): no bank conflicts between the rows of a half warp */ \
        static constexpr int RS = R1 * S + (16 + TPR % 16 - R1 * S % 16) % 16; \
        static constexpr int NZT = (L_ + 4) / 4;  \
    };
PMX_ROW_CFG(32, 8, 4)
PMX_ROW_CFG(48, 8, 6)
PMX_ROW_CFG(64, 8, 8)
PMX_ROW_CFG(96, 8, 12)
PMX_ROW_CFG(128, 16, 8)
PMX_ROW_CFG(192, 16, 12)
PMX_ROW_CFG(256, 32, 8)
PMX_ROW_CFG(384, 32, 12)
PMX_ROW_CFG(512, 32, 16)
#undef PMX_ROW_CFG

__device__ __forceinline__ float2 pick(bool c, float2 a, float2 b) {
    return make_float2(c ? a.x : b.x, c ? a.y : b.y);
}

// Twiddle tables of a length-N transform (float2): w^(b k1) at k1 * R2 + b,
// then the same at b * R1 + k1 (w = exp(-2 pi i / N)).
template <int N>
__device__ __forceinline__ const float2 *tw_fwd(const float2 *tw) { return tw; }
template <int N>
__device__ __forceinline__ const float2 *tw_tr(const float2 *tw) { return tw + N; }

// R1 and R2 of a supported axis length (or half length), on the host.
template <class F>
void mesh_axis_r(int64_t n, F &&f) {
    switch (n) {
        case 64: f(Fac<64>::R1, Fac<64>::R2); break;
        case 96: f(Fac<96>::R1, Fac<96>::R2); break;
        case 128: f(Fac<128>::R1, Fac<128>::R2); break;
        case 192: f(Fac<192>::R1, Fac<192>::R2); break;
        case 256: f(Fac<256>::R1, Fac<256>::R2); break;
        case 384: f(Fac<384>::R1, Fac<384>::R2); break;
        case 512: f(Fac<512>::R1, Fac<512>::R2); break;
        case 768: f(Fac<768>::R1, Fac<768>::R2); break;
        case 1024: f(Fac<1024>::R1, Fac<1024>::R2); break;
    }
}

__device__ __forceinline__ int64_t spec_at(const MeshGeom &g, int64_t x, int ky, int l) {
    return (((x >> 3) * g.n1 + ky) * g.nzt + (l >> 2)) * 32 + (x & 7) * 4 + (l & 3);
}


// Table loads in program order.  Left alone, the compiler hoists all of a
// thread's table loads to the front and spills for their registers: groups of
// GRP keep the latency covered at GRP values.
__device__ __forceinline__ float2 ld_tab2(const float2 *p) {
    float2 v;
    asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
constexpr int GRP = 8;

// buf[at(k)] = v[e] * table[idx(k)] (conjugated for INV), k = reg_freq(e); k = 0 has
// twiddle 1.
template <int R, bool INV, class At, class Idx>
__device__ __forceinline__ void twiddle_store(const float2 (&v)[R], float2 *buf,
                                              const float2 *__restrict__ tw, At &&at, Idx &&idx) {
    static_for<(R + GRP - 1) / GRP>([&](auto G) {
        constexpr int e0 = G * GRP, n = R - e0 < GRP ? R - e0 : GRP;
        float2 w[n];
        static_for<n>([&](auto I) {
            constexpr int k = reg_freq<R>(e0 + I);
            if constexpr (k != 0) w[I] = ld_tab2(tw + idx(k));
        });
        static_for<n>([&](auto I) {
            constexpr int k = reg_freq<R>(e0 + I);
            float2 x = v[e0 + I];
            if constexpr (k != 0) x = INV ? cmulc(x, w[I]) : cmul(x, w[I]);
            buf[at(k)] = x;
        });
    });
}

// Stage 1 of T columns: v holds elements b + a R2 of column t; radix-R1 DFT,
// twiddles, exchange buffer.
template <class C, bool INV>
__device__ __forceinline__ void col_stage1(float2 (&v)[C::R1], float2 *buf, int t, int b,
                                           const float2 *__restrict__ tw) {
    reg_dft<C::R1, INV>(v);
    static_for<C::R1>([&](auto E) {
        constexpr int k1 = reg_freq<C::R1>(E);
        float2 x = v[E];
        if constexpr (k1 != 0) {
            const float2 w = __ldg(tw + k1 * C::R2 + b);
            x = INV ? cmulc(x, w) : cmul(x, w);
        }
        buf[k1 * C::GS + b * C::T + t] = x;
    });
}

// Stage 2 of group (t, k1): u[e] holds frequency k1 + R1 reg_freq(e).
template <class C, bool INV>
__device__ __forceinline__ void col_stage2(float2 (&u)[C::R2], const float2 *buf, int t, int k1) {
#pragma unroll
    for (int b = 0; b < C::R2; ++b) u[b] = buf[k1 * C::GS + b * C::T + t];
    reg_dft<C::R2, INV>(u);
}

// Keeps values parked in shared memory there: without it the compiler forwards
// the stores to the later loads in registers, which costs a block per SM.
__device__ __forceinline__ void parked() { asm volatile("" ::: "memory"); }

// A stride the compiler cannot see through: otherwise the 64-bit offsets of one
// phase's accesses stay in registers (two for each of 32 elements) for the next
// phase that uses the same ones.
__device__ __forceinline__ int64_t fresh(int64_t v) {
    asm volatile("" : "+l"(v));
    return v;
}

// Blocks per SM that `bufs` exchange buffers and `regs` registers per thread
// leave room for.
template <class C>
constexpr int col_blocks(int bufs, int regs) {
    const int by_smem = 227 * 1024 / (bufs * C::BUF * 8 + 1024), by_regs = 65536 / (regs * C::TH);
    const int n = by_smem < by_regs ? by_smem : by_regs;
    return n < 1 ? 1 : n;
}

template <class K>
int smem_opt_in(K *fn, size_t bytes) {
    if (bytes <= 48 * 1024) return PMX_OK;
    PMX_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return PMX_OK;
}
template <class C>
constexpr size_t cols_smem(int bufs) { return (size_t)bufs * C::BUF * sizeof(float2); }

// Calls f(integral_constant<int, N>{}) for the supported length n.
template <class F>
int mesh_axis_dispatch(int64_t n, F &&f) {
    switch (n) {
        case 64: return f(std::integral_constant<int, 64>{});
        case 96: return f(std::integral_constant<int, 96>{});
        case 128: return f(std::integral_constant<int, 128>{});
        case 192: return f(std::integral_constant<int, 192>{});
        case 256: return f(std::integral_constant<int, 256>{});
        case 384: return f(std::integral_constant<int, 384>{});
        case 512: return f(std::integral_constant<int, 512>{});
        case 768: return f(std::integral_constant<int, 768>{});
        case 1024: return f(std::integral_constant<int, 1024>{});
        default: return fail(PMX_ERR_SHAPE, "mesh transform length not supported");
    }
}

}  // namespace pmx
