// x-axis transforms of the Poisson solve, fused with the Green's function and
// the gradients (see pmx_mesh_fft.cuh).

#include <cmath>

#include "pmx_mesh_fft.cuh"

namespace pmx {

namespace {

// Registers per thread of an x kernel.
template <int N>
constexpr int x_regs() { return Fac<N>::R1 >= 24 ? 160 : (Fac<N>::R1 >= 16 ? 96 : 64); }

// The wavenumber tables are read in groups of eight, in program order: left
// alone the compiler hoists all of a thread's table loads to the front, and
// their registers with them.
__device__ __forceinline__ float ld_tab(const float *p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// Inverse first step on a register group in natural order: radix-R2 inverse
// DFT, conjugate twiddles, back into the group's own place in the buffer.
template <int N>
__device__ __forceinline__ void x_inv_step2(const float2 (&w)[Fac<N>::R2], float2 *buf, int t,
                                            int k1, const float2 *__restrict__ twt) {
    using C = XCol<N>;
    float2 u[C::R2];
    reg_natural<C::R2>(w, u);
    reg_dft<C::R2, true>(u);
    twiddle_store<C::R2, true>(u, buf, twt, [&](int b) { return k1 * C::GS + b * C::T + t; },
                               [&](int b) { return b * C::R1 + k1; });
}

// Offset of x = b + A R2 from the column's first block; xbs: 8 x-planes.
template <int R2, int A>
__device__ __forceinline__ int64_t x_off(int b, int64_t xbs) {
    return ((b >> 3) + A * (R2 / 8)) * xbs + (b & 7) * 4;
}

// Inverse second step: radix-R1 inverse DFTs over k1, stored to column t at
// x = b + a R2.
template <int N>
__device__ __forceinline__ void x_inv_step1(const float2 *buf, int t, int b, float2 *dst,
                                            int64_t xbs) {
    using C = XCol<N>;
    float2 v[C::R1];
#pragma unroll
    for (int k1 = 0; k1 < C::R1; ++k1) v[k1] = buf[k1 * C::GS + b * C::T + t];
    reg_dft<C::R1, true>(v);
    const int64_t xs = fresh(xbs);
    static_for<C::R1>([&](auto E) { dst[x_off<C::R2, reg_freq<C::R1>(E)>(b, xs)] = v[E]; });
}

// s0: H in, G_0 out (in place: a block reads its whole tile before it
// writes); s1: Q out.
template <int N>
__global__ void __launch_bounds__(XCol<N>::TH, col_blocks<XCol<N>>(2, x_regs<N>())) k_xaxis_fwd(float2 *s0, float2 *s1,
                                                             const float2 *__restrict__ tw,
                                                             const float *__restrict__ kt,
                                                             const __grid_constant__ GreenTab gt,
                                                             MeshGeom g) {
    using C = XCol<N>;
    constexpr int R1 = C::R1, R2 = C::R2;
    extern __shared__ __align__(16) float2 sm[];
    float2 *A = sm, *B = sm + C::BUF;
    const int nct = (4 * g.nzt + C::T - 1) / C::T;
    const int t = threadIdx.x % C::T, b = threadIdx.x / C::T;
    const int ky = blockIdx.x / nct, l = (blockIdx.x % nct) * C::T + t;
    const bool ok = l < 4 * g.nzt;
    const int64_t xbs = g.n1 * g.nzt * 32;                  // 8 x-planes
    const int64_t at = blockIdx.y * g.unit + ((int64_t)ky * g.nzt + (ok ? l >> 2 : 0)) * 32 + (l & 3);
    float2 *p0 = s0 + at, *p1 = s1 + at;
    after_previous();
    {
        float2 v[R1];
        const int64_t xs = fresh(xbs);
        static_for<R1>([&](auto I) { v[I] = p0[x_off<R2, I>(b, xs)]; });
        col_stage1<C, false>(v, A, t, b, tw_fwd<N>(tw));
    }
    __syncthreads();
    const int64_t tot = g.n0 + g.n1 + g.n2h;
    const float kyj = __ldg(kt + g.n0 + ky), kzl = l < g.n2h ? __ldg(kt + g.n0 + g.n1 + l) : 0.f;
    const float ky2 = __fmul_rn(kyj, kyj), kz2 = __fmul_rn(kzl, kzl);
    const float cc = gt.c[blockIdx.y];
    for (int k1 = b; k1 < R1; k1 += R2) {
        float2 v[R2];
        col_stage2<C, false>(v, A, t, k1);
        float2 w[R2];
        static_for<R2>([&](auto E) {
            const int ix = k1 + R1 * reg_freq<R2>(E);
            const float kxi = ld_tab(kt + ix), mxi = ld_tab(kt + tot + ix);
            const float k2v = __fadd_rn(__fadd_rn(__fmul_rn(kxi, kxi), ky2), kz2);
            // laplace (k = 0 -> 0); c / k^2 to within 2 ulp
            const float rk = k2v != 0.f ? __fdividef(cc, k2v) : 0.f;
            const float pr = -__fmul_rn(v[E].x, rk), pi = -__fmul_rn(v[E].y, rk);
            // P waits in the thread's own group of A while G_0 is transformed
            A[k1 * C::GS + E * C::T + t] = make_float2(pr, pi);
            w[E] = make_float2(__fmul_rn(mxi, pi), -__fmul_rn(mxi, pr));  // -i kx P
            if constexpr (E % 8 == 7) parked();
        });
        x_inv_step2<N>(w, B, t, k1, tw_tr<N>(tw));
        parked();
        static_for<R2>([&](auto E) { v[E] = A[k1 * C::GS + E * C::T + t]; });
        x_inv_step2<N>(v, A, t, k1, tw_tr<N>(tw));
    }
    __syncthreads();
    if (!ok) return;
    x_inv_step1<N>(B, t, b, p0, xbs);
    x_inv_step1<N>(A, t, b, p1, xbs);
}

// s0: C_0 in, S out (in place); s1: D in.
template <int N>
__global__ void __launch_bounds__(XCol<N>::TH, col_blocks<XCol<N>>(2, x_regs<N>())) k_xaxis_adj(float2 *s0, const float2 *s1,
                                                             const float2 *__restrict__ tw,
                                                             const float *__restrict__ kt,
                                                             const __grid_constant__ GreenTab gt,
                                                             MeshGeom g) {
    using C = XCol<N>;
    constexpr int R1 = C::R1, R2 = C::R2;
    extern __shared__ __align__(16) float2 sm[];
    float2 *A = sm, *B = sm + C::BUF;
    const int nct = (4 * g.nzt + C::T - 1) / C::T;
    const int t = threadIdx.x % C::T, b = threadIdx.x / C::T;
    const int ky = blockIdx.x / nct, l = (blockIdx.x % nct) * C::T + t;
    const bool ok = l < 4 * g.nzt;
    const int64_t xbs = g.n1 * g.nzt * 32;
    const int64_t at = blockIdx.y * g.unit + ((int64_t)ky * g.nzt + (ok ? l >> 2 : 0)) * 32 + (l & 3);
    float2 *p0 = s0 + at;
    after_previous();
#pragma unroll 1
    for (int j = 0; j < 2; ++j) {
        const float2 *p = j ? s1 + at : p0;
        float2 v[R1];
        const int64_t xs = fresh(xbs);
        static_for<R1>([&](auto I) { v[I] = p[x_off<R2, I>(b, xs)]; });
        col_stage1<C, false>(v, sm + j * C::BUF, t, b, tw_fwd<N>(tw));
    }
    __syncthreads();
    const int64_t tot = g.n0 + g.n1 + g.n2h;
    const float kyj = __ldg(kt + g.n0 + ky), kzl = l < g.n2h ? __ldg(kt + g.n0 + g.n1 + l) : 0.f;
    const float ky2 = __fmul_rn(kyj, kyj), kz2 = __fmul_rn(kzl, kzl);
    const float cc = gt.c[blockIdx.y];
    for (int k1 = b; k1 < R1; k1 += R2) {
        float2 v[R2];
        col_stage2<C, false>(v, A, t, k1);
        static_for<R2>([&](auto E) { A[k1 * C::GS + E * C::T + t] = v[E]; });
        parked();
        col_stage2<C, false>(v, B, t, k1);
        static_for<R2>([&](auto E) {
            const int ix = k1 + R1 * reg_freq<R2>(E);
            const float kxi = ld_tab(kt + ix), mxi = ld_tab(kt + tot + ix);
            const float k2v = __fadd_rn(__fadd_rn(__fmul_rn(kxi, kxi), ky2), kz2);
            const float2 c0 = A[k1 * C::GS + E * C::T + t];
            const float re = __fadd_rn(-__fmul_rn(mxi, c0.y), v[E].x);
            const float im = __fadd_rn(__fmul_rn(mxi, c0.x), v[E].y);
            const float rk = k2v != 0.f ? __fdividef(cc, k2v) : 0.f;
            v[E] = make_float2(-__fmul_rn(re, rk), -__fmul_rn(im, rk));
            if constexpr (E % 8 == 7) parked();
        });
        x_inv_step2<N>(v, A, t, k1, tw_tr<N>(tw));
    }
    __syncthreads();
    if (!ok) return;
    x_inv_step1<N>(A, t, b, p0, xbs);
}

// Modes in their own layout -> x-inverse-transformed spectra, see mesh_xaxis_modes.
// A tile's p stays in registers where a thread has one group of at most 16 of it;
// else it is read once per spectrum, after the first time from L1 or L2.  256^3: 83
// and 68 us for three and two spectra, 113 and 78 with p read each time.
template <int N>
constexpr bool modes_keep() { return Fac<N>::R1 <= Fac<N>::R2 && Fac<N>::R2 <= 16; }
template <int N>
constexpr int modes_regs() { return modes_keep<N>() || Fac<N>::R1 >= 24 ? 168 : x_regs<N>(); }
template <int N, bool GRADS>
__global__ void __launch_bounds__(XCol<N>::TH, col_blocks<XCol<N>>(1, modes_regs<N>())) k_xaxis_modes(const float2 *__restrict__ modes,
                                                             float scale, float2 *spec,
                                                             const float2 *__restrict__ tw,
                                                             const float *__restrict__ kt,
                                                             MeshGeom g) {
    using C = XCol<N>;
    constexpr int R1 = C::R1, R2 = C::R2;
    extern __shared__ __align__(16) float2 sm[];
    const int nct = (4 * g.nzt + C::T - 1) / C::T;
    const int t = threadIdx.x % C::T, b = threadIdx.x / C::T;
    const int ky = blockIdx.x / nct, l = (blockIdx.x % nct) * C::T + t;
    const bool ok = l < 4 * g.nzt, in = l < g.n2h;
    const int64_t xbs = g.n1 * g.nzt * 32;                  // 8 x-planes
    const int64_t at = ((int64_t)ky * g.nzt + (ok ? l >> 2 : 0)) * 32 + (l & 3);
    after_previous();
    const int64_t tot = g.n0 + g.n1 + g.n2h, xs = g.n1 * g.n2h;
    const float2 *src = modes + (int64_t)ky * g.n2h + l;
    const float kyj = __ldg(kt + g.n0 + ky), kzl = in ? __ldg(kt + g.n0 + g.n1 + l) : 0.f;
    const float ky2 = __fmul_rn(kyj, kyj), kz2 = __fmul_rn(kzl, kzl);
    // p of group k1, in the order of reg_dft
    auto fetch = [&](float2 (&p)[R2], int k1) {
        static_for<R2>([&](auto E) {
            p[E] = in ? src[(k1 + R1 * reg_freq<R2>(E)) * xs] : make_float2(0.f, 0.f);
        });
        static_for<R2>([&](auto E) {
            const float kx = ld_tab(kt + k1 + R1 * reg_freq<R2>(E));
            const float k2 = __fadd_rn(__fadd_rn(__fmul_rn(kx, kx), ky2), kz2);
            const float f = scale * (1.f / k2);   // k = 0 -> 0, whatever the mode
            p[E] = k2 != 0.f ? make_float2(p[E].x * f, p[E].y * f) : make_float2(0.f, 0.f);
        });
    };
    constexpr bool KEEP = modes_keep<N>();
    float2 p[R2];
    if (KEEP && b < R1) fetch(p, b);
#pragma unroll 1
    for (int s = 0; s < (GRADS ? 2 : 3); ++s) {
        for (int k1 = b; k1 < R1; k1 += R2) {
            if (!KEEP) fetch(p, k1);
            float2 w[R2];
            static_for<R2>([&](auto E) {
                const int ix = k1 + R1 * reg_freq<R2>(E);
                const float kx = ld_tab(kt + ix), mx = ld_tab(kt + tot + ix);
                if (GRADS) {
                    w[E] = s == 0 ? make_float2(-(mx * p[E].y), mx * p[E].x)
                                  : make_float2(-p[E].x, -p[E].y);
                } else {
                    const float q = s == 0 ? kx * kx : (s == 1 ? mx : 1.f);
                    w[E] = make_float2(p[E].x * q, p[E].y * q);
                }
            });
            x_inv_step2<N>(w, sm, t, k1, tw_tr<N>(tw));
        }
        __syncthreads();
        if (ok) x_inv_step1<N>(sm, t, b, spec + s * g.unit + at, xbs);
        __syncthreads();
    }
}

__device__ __forceinline__ float2 twiddle(int j, int n) {   // exp(-2 pi i j / n)
    double c, s;
    sincospi(-2.0 * (double)(j % n) / (double)n, &s, &c);
    return make_float2((float)c, (float)s);
}
struct TwAxis {
    int n, R1, R2;
};
__global__ void k_twiddles(TwAxis x, TwAxis y, TwAxis z, float2 *t) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    const TwAxis ax[3] = {x, y, z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int n = ax[a].n;
        if (q >= 0 && q < n) {
            const int k1 = q / ax[a].R2, b = q % ax[a].R2;
            const float2 w = twiddle(k1 * b, n);
            t[q] = w;
            t[n + b * ax[a].R1 + k1] = w;
        }
        q -= n;
        t += 2 * n;
    }
    if (q >= 0 && q <= z.n) t[q] = twiddle(q, 2 * z.n);
}

}  // namespace

int mesh_xaxis_prepare(int64_t n0) {
    return mesh_axis_dispatch(n0, [&](auto N) -> int {
        int st;
        if ((st = smem_opt_in(k_xaxis_fwd<N>, cols_smem<XCol<N>>(2))) ||
            (st = smem_opt_in(k_xaxis_adj<N>, cols_smem<XCol<N>>(2))) ||
            (st = smem_opt_in(k_xaxis_modes<N, false>, cols_smem<XCol<N>>(1))) ||
            (st = smem_opt_in(k_xaxis_modes<N, true>, cols_smem<XCol<N>>(1))))
            return st;
        return PMX_OK;
    });
}

int mesh_xaxis(bool adj, int nslot, const MeshGeom &g, float2 *s0, float2 *s1, const float2 *tw,
               const float *kt, const GreenTab &gt, cudaStream_t st) {
    return mesh_axis_dispatch(g.n0, [&](auto N) -> int {
        using C = XCol<N>;
        const dim3 grid((unsigned)(g.n1 * ((4 * g.nzt + C::T - 1) / C::T)), nslot);
        if (adj)
            PMX_CUDA(launch_after(k_xaxis_adj<N>, grid, C::TH, cols_smem<XCol<N>>(2), st, s0, s1,
                                  tw, kt, gt, g));
        else
            PMX_CUDA(launch_after(k_xaxis_fwd<N>, grid, C::TH, cols_smem<XCol<N>>(2), st, s0, s1,
                                  tw, kt, gt, g));
        PMX_LAUNCH_CHECK("mesh transform, x axis");
        return PMX_OK;
    });
}

int mesh_xaxis_modes(bool grads, const MeshGeom &g, const float2 *modes, float scale, float2 *spec,
                     const float2 *tw, const float *kt, cudaStream_t st) {
    return mesh_axis_dispatch(g.n0, [&](auto N) -> int {
        using C = XCol<N>;
        const unsigned grid = (unsigned)(g.n1 * ((4 * g.nzt + C::T - 1) / C::T));
        const size_t smem = cols_smem<XCol<N>>(1);
        if (grads)
            PMX_CUDA(launch_after(k_xaxis_modes<N, true>, grid, C::TH, smem, st, modes, scale, spec, tw,
                                  kt, g));
        else
            PMX_CUDA(launch_after(k_xaxis_modes<N, false>, grid, C::TH, smem, st, modes, scale, spec, tw,
                                  kt, g));
        PMX_LAUNCH_CHECK("mesh transform of modes, x axis");
        return PMX_OK;
    });
}

int mesh_fft_twiddles_dev(int64_t n0, int64_t n1, int64_t n2, float2 *t, cudaStream_t st) {
    TwAxis ax[3];
    const int64_t n[3] = {n0, n1, n2 / 2};
    for (int a = 0; a < 3; ++a) {
        ax[a].n = (int)n[a];
        if (a < 2)
            mesh_axis_r(n[a], [&](int R1, int R2) { ax[a].R1 = R1; ax[a].R2 = R2; });
        else if (int e = mesh_rows_factors(n2, &ax[a].R1, &ax[a].R2))
            return e;
    }
    const int tot = (int)(n0 + n1 + 2 * n[2] + 1);
    k_twiddles<<<(tot + 63) / 64, 64, 0, st>>>(ax[0], ax[1], ax[2], t);
    PMX_LAUNCH_CHECK("k_twiddles");
    return PMX_OK;
}

// Tables in tw: the x axis' 2 n0 entries, the y axis' 2 n1, then the z axis'
// 2 L and the split's L + 1 (L = n2 / 2); float64 on the host, then float32.
static void axis_table(int64_t n, int R1, int R2, float2 *t) {
    for (int k1 = 0; k1 < R1; ++k1)
        for (int b = 0; b < R2; ++b) {
            const double a = -2.0 * kPi * (double)(b * k1) / (double)n;
            const float2 w = make_float2((float)std::cos(a), (float)std::sin(a));
            t[k1 * R2 + b] = w;
            t[n + b * R1 + k1] = w;
        }
}

bool mesh_fft_supported(int64_t n0, int64_t n1, int64_t n2) {
    for (int64_t n : {n0, n1, n2})
        if (n != 64 && n != 96 && n != 128 && n != 192 && n != 256 && n != 384 && n != 512 &&
            n != 768 && n != 1024)
            return false;
    return true;
}

int64_t mesh_fft_twiddles(int64_t n0, int64_t n1, int64_t n2, float2 *t) {
    const int64_t L = n2 / 2;
    if (t) {
        mesh_axis_r(n0, [&](int R1, int R2) { axis_table(n0, R1, R2, t); });
        mesh_axis_r(n1, [&](int R1, int R2) { axis_table(n1, R1, R2, t + 2 * n0); });
        int R1 = 1, R2 = 1;
        mesh_rows_factors(n2, &R1, &R2);
        axis_table(L, R1, R2, t + 2 * n0 + 2 * n1);
        float2 *s = t + 2 * n0 + 2 * n1 + 2 * L;
        for (int64_t k = 0; k <= L; ++k) {
            const double a = -2.0 * kPi * (double)k / (double)n2;
            s[k] = make_float2((float)std::cos(a), (float)std::sin(a));
        }
    }
    return 2 * n0 + 2 * n1 + 3 * L + 1;
}

}  // namespace pmx
