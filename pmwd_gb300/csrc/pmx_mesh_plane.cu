// z and y axes of the Poisson solve in one kernel (see pmx_mesh_fft.cuh), for planes
// that fit into a block's shared memory.
//
// Forward: the block transforms the z rows of its (y, z) plane, turns them into
// columns in shared memory and writes the y transforms to the spectrum.  Inverse:
// the same backwards.
//
// These sizes live in L2 and are bound by launches and by the latency of a block's
// chain of loads, exchanges and stores: one launch does what two did, and the half
// rows stay in shared memory.  Forward and three inverse planes (us, n^3 meshes):
//          this file       rows and columns
//   n = 64    5.4 +  6.9      9.4 + 24.8 (cuFFT)
//   n = 96    7.7 + 11.6      9.6 + 15.1
//   n = 128  10.4 + 23.8     13.6 + 23.8
//   n = 192  34.5 + 67.5     31.0 + 62.5
// At 192 a plane takes one SM's whole shared memory and nothing overlaps its waits.
// Larger planes in the shared memories of a cluster of 4 or 8 blocks, exchanged
// through them, were slower as well (256: 65 + 161 against 51 + 125; 512: 690 + 1940
// against 385 + 1027).
//
// X[0] and X[L] of a real row are real: they travel as one complex column, which is
// separated after the y transform (and put together before it, from the Hermitian
// parts: the imaginary parts of the two columns after the inverse y transform are
// ignored, as the z transform alone would).

#include "pmx_mesh_fft.cuh"

namespace pmx {

namespace {

template <int N_>
struct PlaneCfg {
    static constexpr int N = N_, L = N / 2;
    using Col = TileCfg<N, L>;
    using Row = RowCfg<L>;
    static constexpr int TH = Col::TH;   // L columns at a time, and N rows
    static constexpr int NG = (Col::R1 + Col::R2 - 1) / Col::R2;   // second-stage groups
    // rows and columns take turns: the values pass through registers in between
    static constexpr int ROWBUF = N * Row::RS, COLBUF = Col::BUF;
    static constexpr int BUF = ROWBUF > COLBUF ? ROWBUF : COLBUF;
    static constexpr size_t SMEM = sizeof(float2) * (BUF + N);     // and column 0
    static_assert(TH == N * Row::TPR && N * L <= BUF && SMEM <= 227 * 1024, "plane split");
};

// Column t of row y within a block's columns: the four rows a warp writes at a time
// fall on different banks.
template <int K>
__device__ __forceinline__ int col_at(int y, int t) {
    if constexpr (K % 32 == 0) t ^= (y & 3) << 3;
    else if constexpr (K % 16 == 0) t ^= (y & 1) << 3;
    return y * K + t;
}

// Real row `src` -> the radix-R2 side of its half-length transform: u0 = group lane, u1 =
// group R1 - lane (R1 / 2 for lane 0).  The row is left filled with `fill`.
template <int L>
__device__ __forceinline__ void row_fwd(float2 *src, float fill, float2 *row, int lane,
                                        const float2 *__restrict__ tw, float2 (&u0)[RowCfg<L>::R2],
                                        float2 (&u1)[RowCfg<L>::R2]) {
    using R = RowCfg<L>;
    constexpr int R1 = R::R1, R2 = R::R2, TPR = R::TPR;
    constexpr int IT = (R2 + TPR - 1) / TPR;
    float2 v[IT][R1];
#pragma unroll
    for (int i = 0; i < IT; ++i)   // every load before the first use
        if (R2 % TPR == 0 || i * TPR + lane < R2) {
#pragma unroll
            for (int a = 0; a < R1; ++a) v[i][a] = __ldcg(src + i * TPR + lane + a * R2);
        }
#pragma unroll
    for (int i = 0; i < IT; ++i)
        if (R2 % TPR == 0 || i * TPR + lane < R2) {
#pragma unroll
            for (int a = 0; a < R1; ++a) src[i * TPR + lane + a * R2] = make_float2(fill, fill);
        }
#pragma unroll
    for (int i = 0; i < IT; ++i) {
        const int b = i * TPR + lane;
        if (R2 % TPR == 0 || b < R2) {
            reg_dft<R1, false>(v[i]);
            static_for<R1>([&](auto E) {
                constexpr int k1 = reg_freq<R1>(E);
                row[k1 * R::S + b] = k1 == 0 ? v[i][E] : cmul(v[i][E], __ldg(tw + k1 * R2 + b));
            });
        }
    }
    __syncwarp();   // a row's threads are in one warp
    const float2 *g0 = row + lane * R::S, *g1 = row + (lane ? R1 - lane : R1 / 2) * R::S;
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

// The pairs (k, L - k) of lane `lane`: k(I), I < R2, as RowPairs of the z kernels.
template <int L, int I>
__device__ __forceinline__ int pair_k(int lane) {
    using R = RowCfg<L>;
    return (2 * I < R::R2 || lane ? lane : R::R1 / 2 - R::R2 / 2 * R::R1) + I * R::R1;
}

// Splits the pairs and hands out(k, X[k]) every column, X[0] and X[L] as one.
template <int L, class Out>
__device__ __forceinline__ void row_split(const float2 (&u0)[RowCfg<L>::R2],
                                          const float2 (&u1)[RowCfg<L>::R2], int lane,
                                          const float2 *__restrict__ twn, Out &&out) {
    constexpr int R2 = RowCfg<L>::R2;
    const bool first = lane == 0;
    static_for<R2>([&](auto I) {
        constexpr int i = I, j = i - R2 / 2;
        float2 zk, zm;
        if constexpr (j < 0) {
            zk = u0[i];
            zm = pick(first, u0[(R2 - i) % R2], u1[R2 - 1 - i]);
        } else {
            zk = pick(first, u1[j], u0[i]);
            zm = pick(first, u1[R2 - 1 - j], u1[R2 - 1 - i]);
        }
        const int k = pair_k<L, i>(lane);
        const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        const float2 o = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
        const float2 wo = cmul(o, __ldg(twn + k));
        const float2 lo = make_float2(e.x + wo.x, e.y + wo.y), hi = make_float2(e.x - wo.x, wo.y - e.y);
        if (i == 0 && first) {
            out(0, make_float2(lo.x, hi.x));
        } else {
            out(k, lo);
            out(L - k, hi);
        }
    });
    if (first) out(L / 2, make_float2(u0[R2 / 2].x, -u0[R2 / 2].y));
}

// Half row in its slot (column 0 holds X[0] and X[L]) -> real row `dst`; the slot is the
// exchange buffer too.
template <int L>
__device__ __forceinline__ void row_inv(float2 *row, float2 *__restrict__ dst, int lane,
                                        const float2 *__restrict__ tw,
                                        const float2 *__restrict__ twn) {
    using R = RowCfg<L>;
    constexpr int R1 = R::R1, R2 = R::R2, TPR = R::TPR;
    const bool first = lane == 0;
    float2 u0[R2], u1[R2];
    {
        float2 p[R2], q[R2];
        static_for<R2>([&](auto I) {
            const int k = pair_k<L, I>(lane);
            p[I] = row[k];
            q[I] = row[I == 0 && first ? 0 : L - k];
        });
        float2 mid = make_float2(0.f, 0.f);
        if (first) {
            mid = row[L / 2];
            mid = make_float2(2.f * mid.x, -2.f * mid.y);
            q[0] = make_float2(p[0].y, 0.f);
            p[0].y = 0.f;
        }
        static_for<R2>([&](auto I) {
            const float2 s = make_float2(p[I].x + q[I].x, p[I].y - q[I].y);
            const float2 d = make_float2(p[I].x - q[I].x, p[I].y + q[I].y);
            const float2 dw = cmulc(d, __ldg(twn + pair_k<L, I>(lane)));
            p[I] = make_float2(s.x - dw.y, s.y + dw.x);
            q[I] = make_float2(s.x + dw.y, dw.x - s.y);
        });
        static_for<R2>([&](auto M) {
            constexpr int m = M, H = R2 / 2;
            if constexpr (m < H) {
                u0[m] = p[m];
                u1[m] = pick(first, p[m + H], q[R2 - 1 - m]);
            } else {
                u0[m] = pick(first, m == H ? mid : q[R2 - m], p[m]);
                u1[m] = pick(first, q[R2 - 1 - m + H], q[R2 - 1 - m]);
            }
        });
    }
    __syncwarp();                                    // the row is read
    const float2 *twt = tw + L;                      // transposed: b R1 + k1
    const int ka = lane, kb = lane ? R1 - lane : R1 / 2;
    reg_dft<R2, true>(u0);
    static_for<R2>([&](auto E) {
        constexpr int b = reg_freq<R2>(E);
        row[ka * R::S + b] = b == 0 ? u0[E] : cmulc(u0[E], __ldg(twt + b * R1 + ka));
    });
    reg_dft<R2, true>(u1);
    static_for<R2>([&](auto E) {
        constexpr int b = reg_freq<R2>(E);
        row[kb * R::S + b] = b == 0 ? u1[E] : cmulc(u1[E], __ldg(twt + b * R1 + kb));
    });
    __syncwarp();
#pragma unroll
    for (int b0 = 0; b0 < R2; b0 += TPR) {
        const int b = b0 + lane;
        if (R2 % TPR == 0 || b < R2) {
            float2 v[R1];
#pragma unroll
            for (int k1 = 0; k1 < R1; ++k1) v[k1] = row[k1 * R::S + b];
            reg_dft<R1, true>(v);
            static_for<R1>([&](auto E) { dst[b + reg_freq<R1>(E) * R2] = v[E]; });
        }
    }
}

// Real planes (slot, x) -> spectra, one per slot.  The planes are left filled with
// `fill`: a mesh that is deposited into again needs no launch for that.
template <int N>
__global__ void __launch_bounds__(PlaneCfg<N>::TH)
k_plane_fwd(float *in, float fill, float2 *__restrict__ spec, const float2 *__restrict__ twy,
            const float2 *__restrict__ twz, MeshGeom g) {
    using P = PlaneCfg<N>;
    using C = typename P::Col;
    using R = typename P::Row;
    constexpr int L = P::L;
    extern __shared__ __align__(16) float2 sm[];
    float2 *zbuf = sm + P::BUF;
    const int64_t p = blockIdx.x;
    after_previous();
    {
        const int y = threadIdx.x / R::TPR, lane = threadIdx.x % R::TPR;
        float2 u0[R::R2], u1[R::R2];
        row_fwd<L>(reinterpret_cast<float2 *>(in) + (p * N + y) * L, fill, sm + y * R::RS, lane,
                   twz, u0, u1);
        __syncthreads();   // the row buffers are read
        row_split<L>(u0, u1, lane, twz + 2 * L,
                     [&](int k, float2 v) { sm[col_at<L>(y, k)] = v; });
    }
    __syncthreads();
    const int t = threadIdx.x % L, b = threadIdx.x / L;
    float2 v[C::R1];
#pragma unroll
    for (int a = 0; a < C::R1; ++a) v[a] = sm[col_at<L>(b + a * C::R2, t)];
    __syncthreads();
    col_stage1<C, false>(v, sm, t, b, twy);
    __syncthreads();
    float2 *dst = spec + (p / g.n0) * g.unit;
    const int64_t x = p % g.n0;
    for (int k1 = b; k1 < C::R1; k1 += C::R2) {
        float2 u[C::R2];
        col_stage2<C, false>(u, sm, t, k1);
        static_for<C::R2>([&](auto E) {
            const int ky = k1 + C::R1 * reg_freq<C::R2>(E);
            if (t == 0) zbuf[ky] = u[E];
            else dst[spec_at(g, x, ky, t)] = u[E];
        });
    }
    __syncthreads();
    for (int ky = threadIdx.x; ky < N; ky += P::TH) {
        const float2 a = zbuf[ky], m = zbuf[ky ? N - ky : 0];
        dst[spec_at(g, x, ky, 0)] = make_float2(0.5f * (a.x + m.x), 0.5f * (a.y - m.y));
        // the columns behind kz = L only fill the last block
        float4 *e = reinterpret_cast<float4 *>(dst + spec_at(g, x, ky, L));
        e[0] = make_float4(0.5f * (a.y + m.y), -0.5f * (a.x - m.x), 0.f, 0.f);
        e[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// Spectra -> real planes: NC = 1, one spectrum per slot; NC = 3, G_0 (spec0) and Q
// (spec1) -> planes (slot, x, j) of the three gradients, one block each.
template <int N, int NC>
__global__ void __launch_bounds__(PlaneCfg<N>::TH)
k_plane_inv(const float2 *__restrict__ spec0, const float2 *__restrict__ spec1,
            float *__restrict__ out, const float2 *__restrict__ twy,
            const float2 *__restrict__ twz, const float *__restrict__ kt, MeshGeom g) {
    using P = PlaneCfg<N>;
    using C = typename P::Col;
    using R = typename P::Row;
    constexpr int L = P::L;
    extern __shared__ __align__(16) float2 sm[];
    const int64_t id = blockIdx.x, p = id / NC;
    const int comp = (int)(id % NC);
    float2 *zbuf = sm + P::BUF;
    const int t = threadIdx.x % L, b = threadIdx.x / L;
    const int64_t x = p % g.n0, slot = p / g.n0, ys = (int64_t)g.nzt * 32;
    const int64_t tot = g.n0 + g.n1 + g.n2h;
    const float *my = kt + tot + g.n0, *mz = my + g.n1;
    const float2 *spec = (NC == 3 && comp ? spec1 : spec0) + slot * g.unit;
    // times -i ky or -i kz: -i k (a + i b) = (k b, -k a)
    auto grad = [&](float2 a, int ky, int kz) {
        if (NC != 3 || comp == 0) return a;
        const float m = comp == 1 ? __ldg(my + ky) : __ldg(mz + kz);
        return make_float2(__fmul_rn(m, a.y), -__fmul_rn(m, a.x));
    };
    after_previous();
    float2 v[C::R1];
    {
        const float2 *src = spec + spec_at(g, x, 0, t);
#pragma unroll
        for (int a = 0; a < C::R1; ++a) v[a] = src[(b + a * C::R2) * ys];
    }
    {
        const float2 *s0 = spec + spec_at(g, x, 0, 0), *sl = spec + spec_at(g, x, 0, L);
        for (int ky = threadIdx.x; ky < N; ky += P::TH) {
            const int km = ky ? N - ky : 0;
            const float2 a = grad(s0[ky * ys], ky, 0), am = grad(s0[km * ys], km, 0);
            const float2 c = grad(sl[ky * ys], ky, L), cm = grad(sl[km * ys], km, L);
            // (a + conj am) / 2 + i (c + conj cm) / 2
            zbuf[ky] = make_float2(0.5f * ((a.x + am.x) - (c.y - cm.y)),
                                   0.5f * ((a.y - am.y) + (c.x + cm.x)));
        }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < C::R1; ++a) {
        const int ky = b + a * C::R2;
        v[a] = t == 0 ? zbuf[ky] : grad(v[a], ky, t);
    }
    col_stage1<C, true>(v, sm, t, b, twy);
    __syncthreads();
    float2 u[P::NG][C::R2];
#pragma unroll
    for (int i = 0; i < P::NG; ++i)
        if (C::R1 % C::R2 == 0 || b + i * C::R2 < C::R1)
            col_stage2<C, true>(u[i], sm, t, b + i * C::R2);
    __syncthreads();   // the columns are in registers
#pragma unroll
    for (int i = 0; i < P::NG; ++i)
        if (C::R1 % C::R2 == 0 || b + i * C::R2 < C::R1)
            static_for<C::R2>([&](auto E) {
                sm[(b + i * C::R2 + C::R1 * reg_freq<C::R2>(E)) * R::RS + t] = u[i][E];
            });
    __syncthreads();
    const int y = threadIdx.x / R::TPR, lane = threadIdx.x % R::TPR;
    row_inv<L>(sm + y * R::RS, reinterpret_cast<float2 *>(out) + (id * N + y) * L, lane, twz,
               twz + 2 * L);
}

template <class F>
int plane_dispatch(int64_t n, F &&f) {
    switch (n) {
        case 64: return f(std::integral_constant<int, 64>{});
        case 96: return f(std::integral_constant<int, 96>{});
        case 128: return f(std::integral_constant<int, 128>{});
        default: return fail(PMX_ERR_SHAPE, "plane transform length not supported");
    }
}

}  // namespace

int mesh_plane_prepare(int64_t n1, int64_t n2, bool *fits) {
    *fits = n1 == n2 && n1 <= 128;
    if (!*fits) return PMX_OK;
    return plane_dispatch(n1, [&](auto N) -> int {
        int st;
        if ((st = smem_opt_in(k_plane_fwd<N>, PlaneCfg<N>::SMEM)) ||
            (st = smem_opt_in(k_plane_inv<N, 1>, PlaneCfg<N>::SMEM)) ||
            (st = smem_opt_in(k_plane_inv<N, 3>, PlaneCfg<N>::SMEM)))
            return st;
        return PMX_OK;
    });
}

int mesh_plane(int kind, int nslot, const MeshGeom &g, float *mesh, float2 *spec0, float2 *spec1,
               const float2 *twy, const float2 *twz, const float *kt, cudaStream_t st) {
    return plane_dispatch(g.n1, [&](auto N) -> int {
        using P = PlaneCfg<N>;
        const unsigned planes = (unsigned)(nslot * g.n0);
        if (kind == MESH_COLS_FWD)
            PMX_CUDA(launch_after(k_plane_fwd<N>, planes, P::TH, P::SMEM, st, mesh, -1.f, spec0,
                                  twy, twz, g));
        else if (kind == MESH_COLS_INV1)
            PMX_CUDA(launch_after(k_plane_inv<N, 1>, planes, P::TH, P::SMEM, st, spec0, nullptr,
                                  mesh, twy, twz, kt, g));
        else
            PMX_CUDA(launch_after(k_plane_inv<N, 3>, 3 * planes, P::TH, P::SMEM, st, spec0, spec1,
                                  mesh, twy, twz, kt, g));
        PMX_LAUNCH_CHECK("mesh transform, z and y axes");
        return PMX_OK;
    });
}

}  // namespace pmx
