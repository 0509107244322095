// z-axis transforms of the Poisson solve (see pmx_mesh_fft.cuh).

#include "pmx_mesh_fft.cuh"

namespace pmx {

namespace {

// A group of 8 half rows passes through shared memory, in blocks of 8 rows x 4
// kz padded to ZB values, on its way to or from global memory, so that it
// moves in whole 256-byte blocks.  Straight from registers it would move in
// 64-byte pieces (2 rows x 4 kz): 1.62 against 1.30 ms for the c2r of 1024
// planes of 1024 x 1024.
constexpr int ZB = 36;

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// Offsets within a nat plane's 8-row group of columns k and L - k of pair i
// (R2 pairs per thread).  Thread 0 pairs k = R1 i with L - R1 i for i < R2 / 2
// and, in the second half, R1 / 2 + R1 j with L minus that (j = i - R2 / 2);
// thread t > 0 pairs k = t + R1 i with L - k.  Each offset is one of four
// per-thread bases plus a constant.
__device__ __forceinline__ int col_off(int k) { return (k >> 2) * ZB + (k & 3); }

template <int L>
struct RowPairs {
    using C = RowCfg<L>;
    static constexpr int STEP = C::R1 / 4 * ZB;   // R1 columns
    int lo0, hi0, lo1, hi1, k0, k1;
    bool first;
    __device__ __forceinline__ explicit RowPairs(int lane) {
        first = lane == 0;
        lo0 = col_off(lane);
        hi0 = col_off(C::R1 - lane);
        k0 = lane;
        lo1 = first ? col_off(C::R1 / 2) - C::R2 / 2 * STEP : lo0;
        hi1 = first ? col_off(C::R1 / 2) + C::R2 / 2 * STEP : hi0;
        k1 = first ? C::R1 / 2 - C::R2 / 2 * C::R1 : lane;
    }
    template <int I>
    __device__ __forceinline__ int lo() const { return (2 * I < C::R2 ? lo0 : lo1) + I * STEP; }
    template <int I>
    __device__ __forceinline__ int hi() const {
        return (2 * I < C::R2 ? hi0 : hi1) + (C::R2 - 1 - I) * STEP;
    }
    template <int I>
    __device__ __forceinline__ int k() const { return (2 * I < C::R2 ? k0 : k1) + I * C::R1; }
};

// Bound: HBM (one read of the real rows, one write of the half rows): 1.43 ms
// for 1024 planes of 1024 x 1024, 6.0 TB/s.  The shared-memory pipe comes next
// (an element crosses shared memory twice); with the split's pairs fetched
// from there as well it bound the kernel at 80% of its rate and 1.62 ms.
template <int L>
__global__ void __launch_bounds__(RowCfg<L>::TH) k_rows_r2c(const float *__restrict__ in,
                                                            float2 *__restrict__ nat,
                                                            const float2 *__restrict__ tw,
                                                            const float2 *__restrict__ twn) {
    using C = RowCfg<L>;
    constexpr int R1 = C::R1, R2 = C::R2, TPR = C::TPR;
    extern __shared__ __align__(16) float2 sm[];
    const int r = threadIdx.x / TPR, lane = threadIdx.x % TPR;
    const int64_t row0 = (int64_t)blockIdx.x * C::ROWS;     // over all planes
    float2 *row = sm + r * C::RS;
    const float2 *src = reinterpret_cast<const float2 *>(in) + (row0 + r) * L;
    constexpr int IT = (R2 + TPR - 1) / TPR;
    float2 v[IT][R1];
    after_previous();
#pragma unroll
    for (int i = 0; i < IT; ++i)   // every load before the first use
        if (R2 % TPR == 0 || i * TPR + lane < R2) {
#pragma unroll
            for (int a = 0; a < R1; ++a) v[i][a] = __ldcs(src + i * TPR + lane + a * R2);
        }
#pragma unroll
    for (int i = 0; i < IT; ++i) {
        const int b = i * TPR + lane;
        if (R2 % TPR == 0 || b < R2) {
            reg_dft<R1, false>(v[i]);
            static_for<R1>([&](auto E) {
                constexpr int k1 = reg_freq<R1>(E);
                row[k1 * C::S + b] = k1 == 0 ? v[i][E] : cmul(v[i][E], __ldg(tw + k1 * R2 + b));
            });
        }
    }
    __syncwarp();   // a row's threads are in one warp
    const RowPairs<L> pr(lane);
    float2 u0[R2], u1[R2];
    {
        const float2 *g0 = row + lane * C::S, *g1 = row + (lane ? R1 - lane : R1 / 2) * C::S;
        float2 t[R2];
#pragma unroll
        for (int c = 0; c < R2; ++c) t[c] = g0[c];
        reg_dft<R2, false>(t);
        reg_natural<R2>(t, u0);
#pragma unroll
        for (int c = 0; c < R2; ++c) t[c] = g1[c];
        reg_dft<R2, false>(t);
        reg_natural<R2>(t, u1);
    }
    // X[k] = E + w^k O, X[L-k] = conj(E - w^k O), E = (Z[k] + conj Z[L-k]) / 2,
    // O = (Z[k] - conj Z[L-k]) / 2i
    __syncthreads();   // the exchange buffer is read
    float2 *dst = sm + (r >> 3) * (C::NZT * ZB) + (r & 7) * 4;
    static_for<R2>([&](auto I) {
        constexpr int i = I, j = i - R2 / 2;
        float2 zk, zm;
        if constexpr (j < 0) {
            zk = u0[i];
            zm = pick(pr.first, u0[(R2 - i) % R2], u1[R2 - 1 - i]);
        } else {
            zk = pick(pr.first, u1[j], u0[i]);
            zm = pick(pr.first, u1[R2 - 1 - j], u1[R2 - 1 - i]);
        }
        const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        const float2 o = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
        const float2 wo = cmul(o, __ldg(twn + pr.template k<i>()));
        dst[pr.template lo<i>()] = make_float2(e.x + wo.x, e.y + wo.y);
        dst[pr.template hi<i>()] = make_float2(e.x - wo.x, wo.y - e.y);
    });
    if (pr.first) dst[col_off(L / 2)] = make_float2(u0[R2 / 2].x, -u0[R2 / 2].y);
    // the columns behind kz = L only fill the last block
    else if (lane < 4) dst[col_off(L + lane)] = make_float2(0.f, 0.f);
    __syncthreads();
    float4 *o = reinterpret_cast<float4 *>(nat + row0 * (4 * C::NZT));
    for (int i = threadIdx.x; i < C::ROWS * 2 * C::NZT; i += C::TH)
        o[i] = *reinterpret_cast<const float4 *>(sm + (i >> 4) * ZB + (i & 15) * 2);
}

template <int L>
__global__ void __launch_bounds__(RowCfg<L>::TH) k_rows_c2r(const float2 *__restrict__ nat,
                                                            float *__restrict__ out,
                                                            const float2 *__restrict__ tw,
                                                            const float2 *__restrict__ twn) {
    using C = RowCfg<L>;
    constexpr int R1 = C::R1, R2 = C::R2, TPR = C::TPR;
    extern __shared__ __align__(16) float2 sm[];
    const int r = threadIdx.x / TPR, lane = threadIdx.x % TPR;
    const int64_t row0 = (int64_t)blockIdx.x * C::ROWS;
    float2 *row = sm + r * C::RS;
    const RowPairs<L> pr(lane);
    float2 u0[R2], u1[R2];
    const float2 *in = nat + row0 * (4 * C::NZT);
    after_previous();
    for (int i = threadIdx.x; i < C::ROWS * 2 * C::NZT; i += C::TH)
        cp_async16(sm + (i >> 4) * ZB + (i & 15) * 2, in + 2 * i);
    cp_async_wait();
    __syncthreads();
    {
        // Zc[k] = S + i w^-k D, Zc[L-k] = conj(S - i w^-k D), S = X[k] + conj X[L-k],
        // D = X[k] - conj X[L-k]; the imaginary parts of X[0] and X[L] are ignored
        const float2 *src = sm + (r >> 3) * (C::NZT * ZB) + (r & 7) * 4;
        float2 p[R2], q[R2];
        static_for<R2>([&](auto I) {
            p[I] = src[pr.template lo<I>()];
            q[I] = src[pr.template hi<I>()];
        });
        float2 mid = make_float2(0.f, 0.f);
        if (pr.first) {
            mid = src[col_off(L / 2)];
            mid = make_float2(2.f * mid.x, -2.f * mid.y);
            p[0].y = 0.f;
            q[0].y = 0.f;
        }
        static_for<R2>([&](auto I) {
            const float2 s = make_float2(p[I].x + q[I].x, p[I].y - q[I].y);
            const float2 d = make_float2(p[I].x - q[I].x, p[I].y + q[I].y);
            const float2 dw = cmulc(d, __ldg(twn + pr.template k<I>()));
            p[I] = make_float2(s.x - dw.y, s.y + dw.x);
            q[I] = make_float2(s.x + dw.y, dw.x - s.y);
        });
        static_for<R2>([&](auto M) {
            constexpr int m = M, H = R2 / 2;
            if constexpr (m < H) {
                u0[m] = p[m];
                u1[m] = pick(pr.first, p[m + H], q[R2 - 1 - m]);
            } else {
                u0[m] = pick(pr.first, m == H ? mid : q[R2 - m], p[m]);
                u1[m] = pick(pr.first, q[R2 - 1 - m + H], q[R2 - 1 - m]);
            }
        });
    }
    {
        __syncthreads();                                    // the staged rows are read
        const float2 *twt = tw + L;                         // transposed: b R1 + k1
        const int ka = lane, kb = lane ? R1 - lane : R1 / 2;
        reg_dft<R2, true>(u0);
        static_for<R2>([&](auto E) {
            constexpr int b = reg_freq<R2>(E);
            row[ka * C::S + b] = b == 0 ? u0[E] : cmulc(u0[E], __ldg(twt + b * R1 + ka));
        });
        reg_dft<R2, true>(u1);
        static_for<R2>([&](auto E) {
            constexpr int b = reg_freq<R2>(E);
            row[kb * C::S + b] = b == 0 ? u1[E] : cmulc(u1[E], __ldg(twt + b * R1 + kb));
        });
    }
    __syncwarp();
    float2 *dst = reinterpret_cast<float2 *>(out) + (row0 + r) * L;
#pragma unroll
    for (int b0 = 0; b0 < R2; b0 += TPR) {
        const int b = b0 + lane;
        if (R2 % TPR == 0 || b < R2) {
            float2 v[R1];
#pragma unroll
            for (int k1 = 0; k1 < R1; ++k1) v[k1] = row[k1 * C::S + b];
            reg_dft<R1, true>(v);
            static_for<R1>([&](auto E) { dst[b + reg_freq<R1>(E) * R2] = v[E]; });
        }
    }
}

template <int L>
constexpr size_t rows_smem() {
    using C = RowCfg<L>;
    const size_t fft = (size_t)C::ROWS * C::RS, st = (size_t)(C::ROWS / 8) * C::NZT * ZB;
    return (st > fft ? st : fft) * sizeof(float2);
}

}  // namespace

int mesh_rows_prepare(int64_t n2) {
    return mesh_axis_dispatch(n2, [&](auto N2) -> int {
        constexpr int L = N2 / 2;
        int st = smem_opt_in(k_rows_r2c<L>, rows_smem<L>());
        return st ? st : smem_opt_in(k_rows_c2r<L>, rows_smem<L>());
    });
}

int mesh_rows_factors(int64_t n2, int *R1, int *R2) {
    return mesh_axis_dispatch(n2, [&](auto N2) -> int {
        *R1 = RowCfg<N2 / 2>::R1;
        *R2 = RowCfg<N2 / 2>::R2;
        return PMX_OK;
    });
}

int mesh_rows(bool inv, const void *in, void *out, const float2 *tw, int64_t planes, int64_t n1,
              int64_t n2, cudaStream_t st) {
    return mesh_axis_dispatch(n2, [&](auto N2) -> int {
        constexpr int L = N2 / 2;
        using C = RowCfg<L>;
        const unsigned grid = (unsigned)(planes * n1 / C::ROWS);
        if (inv)
            PMX_CUDA(launch_after(k_rows_c2r<L>, grid, C::TH, rows_smem<L>(), st,
                                  (const float2 *)in, (float *)out, tw, tw + 2 * L));
        else
            PMX_CUDA(launch_after(k_rows_r2c<L>, grid, C::TH, rows_smem<L>(), st, (const float *)in,
                                  (float2 *)out, tw, tw + 2 * L));
        PMX_LAUNCH_CHECK("mesh transform, z axis");
        return PMX_OK;
    });
}

}  // namespace pmx
