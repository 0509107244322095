// y-axis transforms of the Poisson solve (see pmx_mesh_fft.cuh).

#include "pmx_mesh_fft.cuh"

namespace pmx {

namespace {

// Offset of row y0 + d of a nat plane (column 0), d a constant, and of
// (x, ky, l) of a spectrum.
template <int D>
__device__ __forceinline__ int64_t nat_row(int nzt, int y0) {
    if constexpr (D % 8 == 0)
        return (int64_t)((y0 >> 3) * nzt) * 32 + (y0 & 7) * 4 + (int64_t)(D / 8 * 32) * nzt;
    else
        return (int64_t)(((y0 + D) >> 3) * nzt) * 32 + ((y0 + D) & 7) * 4;
}

// A block's tile: XP x-planes from p (over all slots) times the 4 kz of block
// zt.  Consecutive blocks take the 8 / XP tiles that share 256-byte spec
// blocks, so that L2 merges their pieces.
struct ColTile {
    int64_t p;
    int zt;
    int comp;
};
template <int T>
__device__ __forceinline__ ColTile col_tile(const MeshGeom &g, int ncomp) {
    constexpr int XP = T / 4, PER = 8 / XP;
    const int64_t id = blockIdx.x / PER;
    ColTile c;
    c.comp = (int)(id % ncomp);
    const int64_t q = id / ncomp;
    c.zt = (int)(q % g.nzt);
    c.p = (q / g.nzt) * 8 + (blockIdx.x % PER) * XP;
    return c;
}

// Registers per thread the y kernels are compiled for.  Fewer, and a thread's
// 32 loads are no longer all in flight; more, and too few blocks share an SM.
// At 1024 and 512 points (ms, 1024^3 and 512^3 meshes): three inverse transforms
// 7.6 / 0.70 with 80 registers, 5.3 / 0.51 with 96, 4.8 / 0.50 with 120, 4.9 /
// 0.57 with 168; one forward 1.87 / 0.22, 1.50 / 0.18, 1.62 / 0.17, 1.60 / 0.19.
template <int N>
constexpr int fwd_regs() { return Fac<N>::R1 > 16 ? 96 : 64; }
template <int N>
constexpr int inv_regs() { return N >= 512 ? 120 : fwd_regs<N>(); }
template <int N>
constexpr int adj_regs() { return N > 256 ? 160 : 120; }

// nat planes (slot, x) -> spectra: one per slot.
template <int N>
__global__ void __launch_bounds__(YCol<N>::TH, col_blocks<YCol<N>>(1, fwd_regs<N>()))
k_cols_fwd(const float2 *__restrict__ nat,
           float2 *__restrict__ spec,
           const float2 *__restrict__ tw,
           MeshGeom g) {
    using C = YCol<N>;
    extern __shared__ __align__(16) float2 sm[];
    const ColTile c = col_tile<C::T>(g, 1);
    const int t = threadIdx.x % C::T, b = threadIdx.x / C::T;
    const int xi = t >> 2, l = c.zt * 4 + (t & 3);
    const float2 *src = nat + (c.p + xi) * (g.n1 * 4 * g.nzt) + c.zt * 32 + (t & 3);
    after_previous();
    float2 v[C::R1];
    static_for<C::R1>([&](auto A) { v[A] = src[nat_row<A * C::R2>(g.nzt, b)]; });
    col_stage1<C, false>(v, sm, t, b, tw);
    __syncthreads();
    float2 *dst = spec + (c.p / g.n0) * g.unit;
    const int64_t x = c.p % g.n0 + xi;
    for (int k1 = b; k1 < C::R1; k1 += C::R2) {
        float2 u[C::R2];
        col_stage2<C, false>(u, sm, t, k1);
        static_for<C::R2>([&](auto E) {
            dst[spec_at(g, x, k1 + C::R1 * reg_freq<C::R2>(E), l)] = u[E];
        });
    }
}

// nat planes (slot, x, j) of the three mesh cotangents -> spectra C_0 and D.
template <int N>
__global__ void __launch_bounds__(YCol<N>::TH, col_blocks<YCol<N>>(2, adj_regs<N>()))
k_cols_adj(const float2 *__restrict__ nat,
           float2 *__restrict__ spec0,
           float2 *__restrict__ spec1,
           const float2 *__restrict__ tw,
           const float *__restrict__ kt,
           MeshGeom g) {
    using C = YCol<N>;
    extern __shared__ __align__(16) float2 sm[];
    const ColTile c = col_tile<C::T>(g, 2);
    const int t = threadIdx.x % C::T, b = threadIdx.x / C::T;
    const int xi = t >> 2, l = c.zt * 4 + (t & 3);
    const int64_t ps = g.n1 * 4 * g.nzt;
    const float2 *src = nat + (c.p + xi) * 3 * ps + c.zt * 32 + (t & 3);
    const int64_t x = c.p % g.n0 + xi, slot = c.p / g.n0;
    after_previous();
    float2 v[C::R1];
    if (c.comp == 0) {
        static_for<C::R1>([&](auto A) { v[A] = src[nat_row<A * C::R2>(g.nzt, b)]; });
        col_stage1<C, false>(v, sm, t, b, tw);
        __syncthreads();
            float2 *dst = spec0 + slot * g.unit;
        for (int k1 = b; k1 < C::R1; k1 += C::R2) {
            float2 u[C::R2];
            col_stage2<C, false>(u, sm, t, k1);
            static_for<C::R2>([&](auto E) {
                dst[spec_at(g, x, k1 + C::R1 * reg_freq<C::R2>(E), l)] = u[E];
            });
        }
        return;
    }
    const int64_t tot = g.n0 + g.n1 + g.n2h;
    const float *my = kt + tot + g.n0;
    const float mz = l < g.n2h ? __ldg(kt + tot + g.n0 + g.n1 + l) : 0.f;
    float2 *sm1 = sm + C::BUF;
    // both components' first stages; the second stage of C_1 leaves its
    // result in the thread's own group, where that of C_2 picks it up (adding
    // to values already stored to global memory instead, with one buffer and
    // five blocks per SM, took 6.9 ms at 1024^3 against 5.8)
#pragma unroll 1
    for (int j = 0; j < 2; ++j) {
        const int nzt = (int)fresh(g.nzt);
        static_for<C::R1>([&](auto A) { v[A] = src[(j + 1) * ps + nat_row<A * C::R2>(nzt, b)]; });
        col_stage1<C, false>(v, sm + j * C::BUF, t, b, tw);
    }
    __syncthreads();
    float2 *dst = spec1 + slot * g.unit + spec_at(g, x, 0, l);
    const int64_t ys = fresh((int64_t)g.nzt * 32);
    for (int k1 = b; k1 < C::R1; k1 += C::R2) {
        float2 u[C::R2];
        col_stage2<C, false>(u, sm, t, k1);
        static_for<C::R2>([&](auto E) { sm[k1 * C::GS + E * C::T + t] = u[E]; });
        parked();
        col_stage2<C, false>(u, sm1, t, k1);
        static_for<C::R2>([&](auto E) {
            const int ky = k1 + C::R1 * reg_freq<C::R2>(E);
            const float2 c1 = sm[k1 * C::GS + E * C::T + t];
            const float m1 = __ldg(my + ky);
            // i k (a + i b) = (-k b, k a)
            dst[ky * ys] = make_float2(-__fadd_rn(__fmul_rn(m1, c1.y), __fmul_rn(mz, u[E].y)),
                                       __fadd_rn(__fmul_rn(m1, c1.x), __fmul_rn(mz, u[E].x)));
        });
    }
}

// Spectra -> nat planes: NC = 1, one spectrum per slot; NC = 3, G_0 (spec0)
// and Q (spec1) -> planes (slot, x, j) of the three gradients; NC = 6 (one slot),
// X_2, X_1, X_0 of k_xaxis_modes (spec0) -> planes (x, c) of the second derivatives
// 00 11 22 01 02 12.
template <int N, int NC>
__global__ void __launch_bounds__(YCol<N>::TH, col_blocks<YCol<N>>(1, inv_regs<N>()))
k_cols_inv(const float2 *__restrict__ spec0,
           const float2 *__restrict__ spec1,
           float2 *__restrict__ nat,
           const float2 *__restrict__ tw,
           const float *__restrict__ kt,
           MeshGeom g) {
    using C = YCol<N>;
    extern __shared__ __align__(16) float2 sm[];
    const ColTile c = col_tile<C::T>(g, NC);
    const int t = threadIdx.x % C::T, b = threadIdx.x / C::T;
    const int xi = t >> 2, l = c.zt * 4 + (t & 3);
    const int64_t x = c.p % g.n0 + xi, slot = c.p / g.n0;
    const int64_t tot = g.n0 + g.n1 + g.n2h;
    const float *my = kt + tot + g.n0;
    const float2 *src = (NC == 3 && c.comp ? spec1 : spec0) + slot * g.unit + spec_at(g, x, 0, l);
    if (NC == 6) src += (c.comp == 0 ? 0 : (c.comp == 3 || c.comp == 4 ? 1 : 2)) * g.unit;
    const int64_t ys = (int64_t)g.nzt * 32;
    after_previous();
    float2 v[C::R1];
#pragma unroll
    for (int a = 0; a < C::R1; ++a) v[a] = src[(b + a * C::R2) * ys];
    if (NC == 3 && c.comp == 1) {
#pragma unroll
        for (int a = 0; a < C::R1; ++a) {   // -i k (a + i b) = (k b, -k a)
            const float m = __ldg(my + b + a * C::R2);
            v[a] = make_float2(__fmul_rn(m, v[a].y), -__fmul_rn(m, v[a].x));
        }
    }
    if (NC == 3 && c.comp == 2) {
        const float m = l < g.n2h ? __ldg(kt + tot + g.n0 + g.n1 + l) : 0.f;
#pragma unroll
        for (int a = 0; a < C::R1; ++a) v[a] = make_float2(__fmul_rn(m, v[a].y), -__fmul_rn(m, v[a].x));
    }
    if constexpr (NC == 6) {
        const float *ky = kt + g.n0, *kz = ky + g.n1;
        const float k = l < g.n2h ? __ldg(kz + l) : 0.f, m = l < g.n2h ? __ldg(kz + tot + l) : 0.f;
        const float fz = c.comp == 2 ? k * k : (c.comp >= 4 ? m : 1.f);
        if (c.comp == 1 || c.comp == 3 || c.comp == 5) {
            const float *f = c.comp == 1 ? ky : my;
#pragma unroll
            for (int a = 0; a < C::R1; ++a) {
                const float q = __ldg(f + b + a * C::R2), fy = (c.comp == 1 ? q * q : q) * fz;
                v[a] = make_float2(v[a].x * fy, v[a].y * fy);
            }
        } else {
#pragma unroll
            for (int a = 0; a < C::R1; ++a) v[a] = make_float2(v[a].x * fz, v[a].y * fz);
        }
    }
    col_stage1<C, true>(v, sm, t, b, tw);
    __syncthreads();
    float2 *dst = nat + ((c.p + xi) * NC + c.comp) * (g.n1 * 4 * g.nzt) + c.zt * 32 + (t & 3);
    for (int k1 = b; k1 < C::R1; k1 += C::R2) {
        float2 u[C::R2];
        col_stage2<C, true>(u, sm, t, k1);
        static_for<C::R2>([&](auto E) {
            dst[nat_row<C::R1 * reg_freq<C::R2>(E)>(g.nzt, k1)] = u[E];
        });
    }
}

}  // namespace

int mesh_cols_prepare(int64_t n1) {
    return mesh_axis_dispatch(n1, [&](auto N) -> int {
        int st;
        if ((st = smem_opt_in(k_cols_fwd<N>, cols_smem<YCol<N>>(1))) ||
            (st = smem_opt_in(k_cols_inv<N, 1>, cols_smem<YCol<N>>(1))) ||
            (st = smem_opt_in(k_cols_inv<N, 3>, cols_smem<YCol<N>>(1))) ||
            (st = smem_opt_in(k_cols_inv<N, 6>, cols_smem<YCol<N>>(1))) ||
            (st = smem_opt_in(k_cols_adj<N>, cols_smem<YCol<N>>(2))))
            return st;
        return PMX_OK;
    });
}

int mesh_cols(int kind, int nslot, const MeshGeom &g, float2 *nat, float2 *spec0, float2 *spec1,
              const float2 *tw, const float *kt, cudaStream_t st) {
    return mesh_axis_dispatch(g.n1, [&](auto N) -> int {
        using C = YCol<N>;
        const int64_t tiles = nslot * g.n0 / (C::T / 4) * g.nzt;
        switch (kind) {
            case MESH_COLS_FWD:
                PMX_CUDA(launch_after(k_cols_fwd<N>, (unsigned)tiles, C::TH, cols_smem<YCol<N>>(1),
                                      st, nat, spec0, tw, g));
                break;
            case MESH_COLS_ADJ:
                PMX_CUDA(launch_after(k_cols_adj<N>, (unsigned)(2 * tiles), C::TH,
                                      cols_smem<YCol<N>>(2), st, nat, spec0, spec1, tw, kt, g));
                break;
            case MESH_COLS_INV1:
                PMX_CUDA(launch_after(k_cols_inv<N, 1>, (unsigned)tiles, C::TH,
                                      cols_smem<YCol<N>>(1), st, spec0, nullptr, nat, tw, kt, g));
                break;
            case MESH_COLS_INV6:
                PMX_CUDA(launch_after(k_cols_inv<N, 6>, (unsigned)(6 * tiles), C::TH,
                                      cols_smem<YCol<N>>(1), st, spec0, nullptr, nat, tw, kt, g));
                break;
            default:
                PMX_CUDA(launch_after(k_cols_inv<N, 3>, (unsigned)(3 * tiles), C::TH,
                                      cols_smem<YCol<N>>(1), st, spec0, spec1, nat, tw, kt, g));
        }
        PMX_LAUNCH_CHECK("mesh transform, y axis");
        return PMX_OK;
    });
}

}  // namespace pmx
