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

// The y kernels' block order: eight consecutive x-planes of one column tile,
// so that the 32-byte pieces of a spectrum block are touched together.
struct ColTile {
    int64_t p;   // plane (over all slots)
    int l0;      // first column
    int comp;
};
template <int T>
__device__ __forceinline__ ColTile col_tile(const MeshGeom &g, int ncomp) {
    const int nct = (4 * g.nzt + T - 1) / T;
    const int64_t id = blockIdx.x >> 3;
    ColTile c;
    c.comp = (int)(id % ncomp);
    const int64_t q = id / ncomp;
    c.l0 = (int)(q % nct) * T;
    c.p = (q / nct) * 8 + (blockIdx.x & 7);
    return c;
}

// nat planes (slot, x) -> spectra: one per slot.
template <int N>
__global__ void __launch_bounds__(ColCfg<N>::TH, col_blocks<N>(1) > 5 ? 5 : col_blocks<N>(1)) k_cols_fwd(const float2 *__restrict__ nat,
                                                            float2 *__restrict__ spec,
                                                            const float2 *__restrict__ tw,
                                                            MeshGeom g) {
    using C = ColCfg<N>;
    extern __shared__ __align__(16) float2 sm[];
    const ColTile c = col_tile<C::T>(g, 1);
    const int t = threadIdx.x % C::T, b = threadIdx.x / C::T, l = c.l0 + t;
    const bool ok = l < 4 * g.nzt;
    const float2 *src = nat + c.p * (g.n1 * 4 * g.nzt) + (ok ? l >> 2 : 0) * 32 + (l & 3);
    float2 v[C::R1];
    static_for<C::R1>([&](auto A) { v[A] = src[nat_row<A * C::R2>(g.nzt, b)]; });
    col_stage1<N, false>(v, sm, t, b, tw);
    __syncthreads();
    if (!ok) return;
    float2 *dst = spec + (c.p / g.n0) * g.unit;
    const int64_t x = c.p % g.n0;
    for (int k1 = b; k1 < C::R1; k1 += C::R2) {
        float2 u[C::R2];
        col_stage2<N, false>(u, sm, t, k1);
        static_for<C::R2>([&](auto E) {
            dst[spec_at(g, x, k1 + C::R1 * reg_freq<C::R2>(E), l)] = u[E];
        });
    }
}

// nat planes (slot, x, j) of the three mesh cotangents -> spectra C_0 and D.
template <int N>
__global__ void __launch_bounds__(ColCfg<N>::TH, col_blocks<N>(2)) k_cols_adj(const float2 *__restrict__ nat,
                                                            float2 *__restrict__ spec0,
                                                            float2 *__restrict__ spec1,
                                                            const float2 *__restrict__ tw,
                                                            const float *__restrict__ kt,
                                                            MeshGeom g) {
    using C = ColCfg<N>;
    extern __shared__ __align__(16) float2 sm[];
    const ColTile c = col_tile<C::T>(g, 2);
    const int t = threadIdx.x % C::T, b = threadIdx.x / C::T, l = c.l0 + t;
    const bool ok = l < 4 * g.nzt;
    const int64_t ps = g.n1 * 4 * g.nzt;
    const float2 *src = nat + c.p * 3 * ps + (ok ? l >> 2 : 0) * 32 + (l & 3);
    const int64_t x = c.p % g.n0, slot = c.p / g.n0;
    float2 v[C::R1];
    if (c.comp == 0) {
        static_for<C::R1>([&](auto A) { v[A] = src[nat_row<A * C::R2>(g.nzt, b)]; });
        col_stage1<N, false>(v, sm, t, b, tw);
        __syncthreads();
        if (!ok) return;
        float2 *dst = spec0 + slot * g.unit;
        for (int k1 = b; k1 < C::R1; k1 += C::R2) {
            float2 u[C::R2];
            col_stage2<N, false>(u, sm, t, k1);
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
    // result in the thread's own group, where that of C_2 picks it up
#pragma unroll 1
    for (int j = 0; j < 2; ++j) {
        static_for<C::R1>([&](auto A) { v[A] = src[(j + 1) * ps + nat_row<A * C::R2>(g.nzt, b)]; });
        col_stage1<N, false>(v, sm + j * C::BUF, t, b, tw);
    }
    __syncthreads();
    if (!ok) return;
    float2 *dst = spec1 + slot * g.unit;
    for (int k1 = b; k1 < C::R1; k1 += C::R2) {
        float2 u[C::R2];
        col_stage2<N, false>(u, sm, t, k1);
        static_for<C::R2>([&](auto E) { sm[k1 * C::GS + E * C::T + t] = u[E]; });
        parked();
        col_stage2<N, false>(u, sm1, t, k1);
        static_for<C::R2>([&](auto E) {
            const int ky = k1 + C::R1 * reg_freq<C::R2>(E);
            const float2 c1 = sm[k1 * C::GS + E * C::T + t];
            const float m1 = __ldg(my + ky);
            // i k (a + i b) = (-k b, k a)
            dst[spec_at(g, x, ky, l)] =
                make_float2(-__fadd_rn(__fmul_rn(m1, c1.y), __fmul_rn(mz, u[E].y)),
                            __fadd_rn(__fmul_rn(m1, c1.x), __fmul_rn(mz, u[E].x)));
        });
    }
}

// Spectra -> nat planes: NC = 1, one spectrum per slot; NC = 3, G_0 (spec0)
// and Q (spec1) -> planes (slot, x, j) of the three gradients.
template <int N, int NC>
__global__ void __launch_bounds__(ColCfg<N>::TH, col_blocks<N>(1) > 5 ? 5 : col_blocks<N>(1)) k_cols_inv(const float2 *__restrict__ spec0,
                                                            const float2 *__restrict__ spec1,
                                                            float2 *__restrict__ nat,
                                                            const float2 *__restrict__ tw,
                                                            const float *__restrict__ kt,
                                                            MeshGeom g) {
    using C = ColCfg<N>;
    extern __shared__ __align__(16) float2 sm[];
    const ColTile c = col_tile<C::T>(g, NC);
    const int t = threadIdx.x % C::T, b = threadIdx.x / C::T, l = c.l0 + t;
    const bool ok = l < 4 * g.nzt;
    const int64_t x = c.p % g.n0, slot = c.p / g.n0;
    const int64_t tot = g.n0 + g.n1 + g.n2h;
    const float *my = kt + tot + g.n0;
    const float2 *src = (NC == 3 && c.comp ? spec1 : spec0) + slot * g.unit + spec_at(g, x, 0, ok ? l : 0);
    const int64_t ys = (int64_t)g.nzt * 32;
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
    col_stage1<N, true>(v, sm, t, b, tw);
    __syncthreads();
    if (!ok) return;
    float2 *dst = nat + (c.p * NC + c.comp) * (g.n1 * 4 * g.nzt) + (l >> 2) * 32 + (l & 3);
    for (int k1 = b; k1 < C::R1; k1 += C::R2) {
        float2 u[C::R2];
        col_stage2<N, true>(u, sm, t, k1);
        static_for<C::R2>([&](auto E) {
            dst[nat_row<C::R1 * reg_freq<C::R2>(E)>(g.nzt, k1)] = u[E];
        });
    }
}

}  // namespace

int mesh_cols_prepare(int64_t n1) {
    return mesh_axis_dispatch(n1, [&](auto N) -> int {
        int st;
        if ((st = smem_opt_in(k_cols_fwd<N>, cols_smem<N>(1))) ||
            (st = smem_opt_in(k_cols_inv<N, 1>, cols_smem<N>(1))) ||
            (st = smem_opt_in(k_cols_inv<N, 3>, cols_smem<N>(1))) ||
            (st = smem_opt_in(k_cols_adj<N>, cols_smem<N>(2))))
            return st;
        return PMX_OK;
    });
}

int mesh_cols(int kind, int nslot, const MeshGeom &g, float2 *nat, float2 *spec0, float2 *spec1,
              const float2 *tw, const float *kt, cudaStream_t st) {
    return mesh_axis_dispatch(g.n1, [&](auto N) -> int {
        using C = ColCfg<N>;
        const int64_t tiles = nslot * g.n0 * ((4 * g.nzt + C::T - 1) / C::T);
        switch (kind) {
            case MESH_COLS_FWD:
                k_cols_fwd<N><<<(unsigned)tiles, C::TH, cols_smem<N>(1), st>>>(nat, spec0, tw, g);
                break;
            case MESH_COLS_ADJ:
                k_cols_adj<N><<<(unsigned)(2 * tiles), C::TH, cols_smem<N>(2), st>>>(nat, spec0, spec1,
                                                                                     tw, kt, g);
                break;
            case MESH_COLS_INV1:
                k_cols_inv<N, 1><<<(unsigned)tiles, C::TH, cols_smem<N>(1), st>>>(spec0, nullptr, nat,
                                                                                  tw, kt, g);
                break;
            default:
                k_cols_inv<N, 3><<<(unsigned)(3 * tiles), C::TH, cols_smem<N>(1), st>>>(spec0, spec1,
                                                                                        nat, tw, kt, g);
        }
        PMX_LAUNCH_CHECK("mesh transform, y axis");
        return PMX_OK;
    });
}

}  // namespace pmx
