// Lagrangian perturbation theory (pmwd/lpt.py:13-76, 136-212) on a 3-D grid:
// the Fourier- and real-space stages between the caller's transforms, and
// their transposes.
//
//   modes --k_lpt_strain--> six strain spectra  --c2r--> phi
//   phi   --k_lpt_source--> 2nd-order source L  --r2c--> src2
//   modes, src2 --k_lpt_grad--> -i k of both potentials  --c2r--> g
//   g     --k_lpt_disp--> pmid, disp, vel
//
// Each stage reads its inputs once and writes its outputs once (HBM is the
// bound).  As separate tensor operations the same stages took about 110 launches
// and 2.4 of 3.6 ms at 256^3.  Transforms are unnormalised; 1 / N is applied
// where a stage reads their result.
//
// pmx_lpt_solve does all of it with the transforms of pmx_mesh_fft.cuh where they
// have the shape: ky and kz are constant along x, so the x axis makes three spectra
// of the modes for the six strains (of kx^2 p, kx p, p) and two for the three
// gradients, and the spectra between the axes are never written in full.  256^3:
// 0.95 ms of device time against 1.60 with 3-D cuFFT between the stages.

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "pmx_internal.cuh"

using namespace pmx;

#define PMX_ALIGNED(bytes, ...) \
    if (!aligned(bytes, __VA_ARGS__)) return fail(PMX_ERR_ALIGN, "arrays must be on " #bytes " bytes")

namespace {

constexpr int LT = 256;

// Tables of one grid, in one float array: k of the three axes (n0 + n1 + n2h),
// the same with the Nyquist entries zeroed (lpt.py:24-30, gravity.py:40-43),
// the lattice displacements (n0 + n1 + n2), then the lattice pmid as int16.
struct LptGrid {
    int n0, n1, n2, n2h;
    const float *tab;
    __device__ const float *k(int a) const { return tab + (a > 0 ? n0 : 0) + (a > 1 ? n1 : 0); }
    __device__ const float *kz(int a) const { return k(a) + n0 + n1 + n2h; }
    __device__ const float *lat(int a) const {
        return tab + 2 * (n0 + n1 + n2h) + (a > 0 ? n0 : 0) + (a > 1 ? n1 : 0);
    }
    __device__ const int16_t *pm(int a) const {
        return reinterpret_cast<const int16_t *>(tab + 2 * (n0 + n1 + n2h) + n0 + n1 + n2) +
               (a > 0 ? n0 : 0) + (a > 1 ? n1 : 0);
    }
};

int64_t table_floats(int n0, int n1, int n2) {
    return 2 * (int64_t)(n0 + n1 + n2 / 2 + 1) + (n0 + n1 + n2) + (n0 + n1 + n2 + 1) / 2;
}

struct LptTables {
    int n[3], mesh[3];
    double period;     // 2 pi / ptcl_spacing
    float nyq, eps;
    double unit[3];    // cell_size / n
    float *tab;
};

// float64, as numpy's fftfreq (i * (1 / n)) and the lattice of
// particles.py:109-154 compute them.
__global__ void k_lpt_tables(LptTables t) {
    const int n2h = t.n[2] / 2 + 1, nk = t.n[0] + t.n[1] + n2h, nl = t.n[0] + t.n[1] + t.n[2];
    float *lat = t.tab + 2 * nk;
    int16_t *pm = reinterpret_cast<int16_t *>(lat + nl);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nk + nl; q += gridDim.x * blockDim.x) {
        if (q < nk) {
            const int a = q < t.n[0] ? 0 : (q < t.n[0] + t.n[1] ? 1 : 2), n = t.n[a];
            const int i = q - (a > 0 ? t.n[0] : 0) - (a > 1 ? t.n[1] : 0);
            const int f = a == 2 || i < (n + 1) / 2 ? i : i - n;
            const float k = (float)__dmul_rn(__dmul_rn((double)f, __ddiv_rn(1.0, (double)n)), t.period);
            t.tab[q] = k;
            t.tab[nk + q] = fabsf(__fsub_rn(fabsf(k), t.nyq)) <= t.eps ? 0.f : k;
        } else {
            const int p = q - nk, a = p < t.n[0] ? 0 : (p < t.n[0] + t.n[1] ? 1 : 2), n = t.n[a];
            const int i = p - (a > 0 ? t.n[0] : 0) - (a > 1 ? t.n[1] : 0);
            const double r = rint(__dmul_rn((double)t.mesh[a], __ddiv_rn((double)i, (double)n)));
            pm[p] = (int16_t)(int)r;
            lat[p] = (float)__dmul_rn((double)((int64_t)i * t.mesh[a] - (int64_t)r * n), t.unit[a]);
        }
    }
}

// Iteration over the half spectrum: a warp per (a, b) row, the lanes along the
// axis that is contiguous in memory; ax[] names the axes (0, 1, 2) of a, b, c.
struct Walk {
    int n[3], ax[3];
    int64_t st[3];   // strides of the strided spectra, per axis 0, 1, 2
    int64_t batch;   // stride from one of their spectra to the next
};

template <class F>
__device__ __forceinline__ void walk(const Walk &w, F &&f) {
    const int lane = threadIdx.x & 31;
    const int64_t rows = (int64_t)w.n[0] * w.n[1], nw = (int64_t)gridDim.x * (LT / 32);
    for (int64_t r = (int64_t)blockIdx.x * (LT / 32) + (threadIdx.x >> 5); r < rows; r += nw) {
        const int a = (int)(r / w.n[1]), b = (int)(r - (int64_t)a * w.n[1]);
        int i[3];
        i[w.ax[0]] = a;
        i[w.ax[1]] = b;
        for (int c = lane; c < w.n[2]; c += 32) {
            i[w.ax[2]] = c;
            f(i[0], i[1], i[2], i[0] * w.st[0] + i[1] * w.st[1] + i[2] * w.st[2]);
        }
    }
}

__device__ __forceinline__ float inv_k2(float kx, float ky, float kz) {
    const float k2 = __fadd_rn(__fadd_rn(__fmul_rn(kx, kx), __fmul_rn(ky, ky)), __fmul_rn(kz, kz));
    return k2 != 0.f ? -1.f / k2 : 0.f;
}
__device__ __forceinline__ float2 scale2(float2 v, float s) { return make_float2(v.x * s, v.y * s); }
// v times a multiple s of inv_k2: 0 where that is, also of an infinite or NaN v (the k = 0
// mode of a spectrum like 1 / k).
__device__ __forceinline__ float2 solve2(float2 v, float s) {
    return s != 0.f ? scale2(v, s) : make_float2(0.f, 0.f);
}

// out[c] = -k_i k_j pot, pot = -scale modes / k^2, pairs 00 11 22 01 02 12; the
// Nyquist entries count only on the diagonal (lpt.py:13-37).
__global__ void __launch_bounds__(LT) k_lpt_strain(const float2 *__restrict__ modes,
                                                   float2 *__restrict__ out, LptGrid g, Walk w,
                                                   float scale) {
    walk(w, [&](int i, int j, int l, int64_t o) {
        const float kx = __ldg(g.k(0) + i), ky = __ldg(g.k(1) + j), kz = __ldg(g.k(2) + l);
        const float mx = __ldg(g.kz(0) + i), my = __ldg(g.kz(1) + j), mz = __ldg(g.kz(2) + l);
        const float2 p = solve2(modes[o], -scale * inv_k2(kx, ky, kz));   // -pot
        out[o] = scale2(p, kx * kx);
        out[o + w.batch] = scale2(p, ky * ky);
        out[o + 2 * w.batch] = scale2(p, kz * kz);
        out[o + 3 * w.batch] = scale2(p, mx * my);
        out[o + 4 * w.batch] = scale2(p, mx * mz);
        out[o + 5 * w.batch] = scale2(p, my * mz);
    });
}

// Fields of a real grid: element r of x-plane x of field c at x xs + c cs + r.
struct Fields {
    int64_t xs, cs;
};

// L = phi_00 phi_22 + phi_00 phi_11 + phi_11 phi_22 - phi_01^2 - phi_02^2 - phi_12^2
// (lpt.py:40-76), phi = s times the transforms.  A block row per x-plane of pl
// values, V at a time.
__device__ __forceinline__ float lpt_source(const float (&p)[6]) {
    float v = fmaf(p[0], p[1], p[0] * p[2]);
    v = fmaf(p[1], p[2], v);
#pragma unroll
    for (int c = 3; c < 6; ++c) v = fmaf(-p[c], p[c], v);
    return v;
}
template <int V>
__global__ void __launch_bounds__(LT) k_lpt_source(const float *__restrict__ phi,
                                                   float *__restrict__ L, int64_t pl, int64_t n0,
                                                   Fields f, float s) {
    after_previous();
    for (int64_t x = blockIdx.y; x < n0; x += gridDim.y) {
        const float *ph = phi + x * f.xs;
        for (int64_t q = (blockIdx.x * (int64_t)LT + threadIdx.x) * V; q < pl;
             q += (int64_t)gridDim.x * LT * V) {
            if constexpr (V == 4) {
                float4 u[6];
#pragma unroll
                for (int c = 0; c < 6; ++c)
                    u[c] = *reinterpret_cast<const float4 *>(ph + q + c * f.cs);
                float o[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float p[6];
#pragma unroll
                    for (int c = 0; c < 6; ++c) p[c] = s * (&u[c].x)[i];
                    o[i] = lpt_source(p);
                }
                *reinterpret_cast<float4 *>(L + x * pl + q) = make_float4(o[0], o[1], o[2], o[3]);
            } else {
                float p[6];
#pragma unroll
                for (int c = 0; c < 6; ++c) p[c] = s * ph[q + c * f.cs];
                L[x * pl + q] = lpt_source(p);
            }
        }
    }
}

// out[3 o + a] = -i k_a pot_o, pot_0 = -scale modes / k^2, pot_1 = -src2 / k^2
// (src2 NULL: first order only); modes and out share the walk's strides, src2
// has its own.
__global__ void __launch_bounds__(LT) k_lpt_grad(const float2 *__restrict__ modes,
                                                 const float2 *__restrict__ src2, int64_t s0,
                                                 int64_t s1, int64_t s2, float2 *__restrict__ out,
                                                 LptGrid g, Walk w, float scale) {
    walk(w, [&](int i, int j, int l, int64_t o) {
        const float ik = inv_k2(__ldg(g.k(0) + i), __ldg(g.k(1) + j), __ldg(g.k(2) + l));
        const float m[3] = {__ldg(g.kz(0) + i), __ldg(g.kz(1) + j), __ldg(g.kz(2) + l)};
        const float2 p = solve2(modes[o], scale * ik);
#pragma unroll
        for (int a = 0; a < 3; ++a)   // (-i k)(x + i y) = (k y, -k x)
            out[o + a * w.batch] = make_float2(m[a] * p.y, -(m[a] * p.x));
        if (src2) {
            const float2 q = solve2(src2[i * s0 + j * s1 + l * s2], ik);
#pragma unroll
            for (int a = 0; a < 3; ++a)
                out[o + (3 + a) * w.batch] = make_float2(m[a] * q.y, -(m[a] * q.x));
        }
    });
}

struct LptFac {
    float f[4];         // D_1, a^2 H dD_1/dlna, D_2, a^2 H dD_2/dlna
    const float *dev;   // or in device memory (a graph's input)
};

constexpr int LPT_PB = 2;

// pmid and disp of the lattice plus disp += D_m g_m, vel += a^2 H dD_m/dlna g_m
// order by order (lpt.py:197-210); g = s times the transforms, those of order 2 at
// gr2.  The bound is HBM (54 bytes per particle: 0.13 ms at
// 256^3), given enough loads in flight: a thread fetches two particles' fields
// before it uses the first, and the outputs pass through shared memory so that a
// warp stores whole lines.  0.136 ms; one particle per thread 0.22, with three
// 12-byte-strided stores each 0.25.
__global__ void __launch_bounds__(LT) k_lpt_disp(const float *__restrict__ gr,
                                                 const float *__restrict__ gr2, Fields fl, int orders,
                                                 int16_t *__restrict__ pmid,
                                                 float *__restrict__ disp, float *__restrict__ vel,
                                                 LptGrid g, LptFac f, float s) {
    after_previous();
    constexpr int PB = LPT_PB * LT;   // particles of a block's turn
    __shared__ __align__(16) float sd[3 * PB], sv[3 * PB];
    __shared__ __align__(16) int16_t sp[3 * PB];
    // whole turns are stored in 16-byte pieces (3 PB values of either type are)
    const bool wide = (((uintptr_t)pmid | (uintptr_t)disp | (uintptr_t)vel) & 15) == 0;
    const int64_t pl = (int64_t)g.n1 * g.n2, n = g.n0 * pl;
    float fac[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) fac[u] = s * (f.dev ? (u < 2 * orders ? f.dev[u] : 0.f) : f.f[u]);
    for (int64_t q0 = blockIdx.x * (int64_t)PB; q0 < n; q0 += (int64_t)gridDim.x * PB) {
        int c[LPT_PB][3];
        float x[LPT_PB][2][3];
#pragma unroll
        for (int i = 0; i < LPT_PB; ++i) {   // every load before the first use
            const int64_t q = q0 + i * LT + threadIdx.x < n ? q0 + i * LT + threadIdx.x : n - 1;
            if (n <= 0x7fffffff) {   // 32-bit divisions
                const unsigned u = (unsigned)q / (unsigned)g.n2;
                c[i][2] = (int)((unsigned)q - u * (unsigned)g.n2);
                c[i][0] = (int)(u / (unsigned)g.n1);
                c[i][1] = (int)(u - (unsigned)c[i][0] * (unsigned)g.n1);
            } else {
                const int64_t r = q / g.n2;
                c[i][2] = (int)(q - r * g.n2);
                c[i][0] = (int)(r / g.n1);
                c[i][1] = (int)(r - (int64_t)c[i][0] * g.n1);
            }
            const int64_t at = c[i][0] * fl.xs + ((int64_t)c[i][1] * g.n2 + c[i][2]);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                x[i][0][a] = gr[at + a * fl.cs];
                x[i][1][a] = orders > 1 ? gr2[at + a * fl.cs] : 0.f;
            }
        }
#pragma unroll
        for (int i = 0; i < LPT_PB; ++i)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const int o = 3 * (i * LT + threadIdx.x) + a;
                float d = fmaf(fac[0], x[i][0][a], __ldg(g.lat(a) + c[i][a]));
                float v = fac[1] * x[i][0][a];
                if (orders > 1) {
                    d = fmaf(fac[2], x[i][1][a], d);
                    v = fmaf(fac[3], x[i][1][a], v);
                }
                sp[o] = g.pm(a)[c[i][a]];
                sd[o] = d;
                sv[o] = v;
            }
        __syncthreads();
        const int m = 3 * (int)(n - q0 < PB ? n - q0 : PB);
        if (wide && m == 3 * PB) {
            for (int i = threadIdx.x; i < 3 * PB / 4; i += LT) {
                reinterpret_cast<float4 *>(disp + 3 * q0)[i] = reinterpret_cast<float4 *>(sd)[i];
                reinterpret_cast<float4 *>(vel + 3 * q0)[i] = reinterpret_cast<float4 *>(sv)[i];
            }
            for (int i = threadIdx.x; i < 3 * PB / 8; i += LT)
                reinterpret_cast<int4 *>(pmid + 3 * q0)[i] = reinterpret_cast<int4 *>(sp)[i];
        } else {
            for (int i = threadIdx.x; i < m; i += LT) {
                pmid[3 * q0 + i] = sp[i];
                disp[3 * q0 + i] = sd[i];
                vel[3 * q0 + i] = sv[i];
            }
        }
        __syncthreads();
    }
}

// Transpose of k_lpt_disp: out[3 o + a] = D_o disp_cot_a + V_o vel_cot_a.
__global__ void __launch_bounds__(LT) k_lpt_disp_adj(const float *__restrict__ dc,
                                                     const float *__restrict__ vc, int orders,
                                                     float *__restrict__ out, int64_t n, LptFac f) {
    for (int64_t q = blockIdx.x * (int64_t)LT + threadIdx.x; q < n; q += (int64_t)gridDim.x * LT) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float d = dc[3 * q + a], v = vc[3 * q + a];
#pragma unroll
            for (int o = 0; o < 2; ++o)
                if (o < orders) out[q + (3 * o + a) * n] = fmaf(f.f[2 * o + 1], v, f.f[2 * o] * d);
        }
    }
}

// The source's cotangent in Fourier space, divided by the multiplicity that the
// transposed r2c and c2r bring and take away: out = -(s / k^2) sum_a i k_a C_a.
__global__ void __launch_bounds__(LT) k_lpt_src_adj(const float2 *__restrict__ C,
                                                    float2 *__restrict__ out, LptGrid g, Walk w,
                                                    float s) {
    walk(w, [&](int i, int j, int l, int64_t o) {
        const float ik = s * inv_k2(__ldg(g.k(0) + i), __ldg(g.k(1) + j), __ldg(g.k(2) + l));
        const float m[3] = {__ldg(g.kz(0) + i), __ldg(g.kz(1) + j), __ldg(g.kz(2) + l)};
        float re = 0.f, im = 0.f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {   // i k (x + i y) = (-k y, k x)
            const float2 c = C[o + a * w.batch];
            re = fmaf(-m[a], c.y, re);
            im = fmaf(m[a], c.x, im);
        }
        out[((int64_t)i * g.n1 + j) * g.n2h + l] = solve2(make_float2(re, im), ik);
    });
}

// Cotangents of the six strains: out_c = Lc dL / dphi_c, phi = s times the
// transforms.
__global__ void __launch_bounds__(LT) k_lpt_source_adj(const float *__restrict__ phi,
                                                       const float *__restrict__ Lc,
                                                       float *__restrict__ out, int64_t n, float s) {
    for (int64_t q = blockIdx.x * (int64_t)LT + threadIdx.x; q < n; q += (int64_t)gridDim.x * LT) {
        float p[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) p[c] = s * phi[q + c * n];
        const float t = Lc[q];
        out[q] = t * (p[1] + p[2]);
        out[q + n] = t * (p[0] + p[2]);
        out[q + 2 * n] = t * (p[0] + p[1]);
#pragma unroll
        for (int c = 3; c < 6; ++c) out[q + c * n] = -2.f * t * p[c];
    }
}

// Cotangent of the modes: w s scale (-1 / k^2) [ sum_a i k_a C_a - sum_ij k_i k_j S_ij ],
// w the number of modes a half-spectrum entry stands for (S NULL: first order).
__global__ void __launch_bounds__(LT) k_lpt_modes_adj(const float2 *__restrict__ C,
                                                      const float2 *__restrict__ S,
                                                      float2 *__restrict__ out, int64_t s0,
                                                      int64_t s1, int64_t s2, LptGrid g, Walk w,
                                                      float s) {
    walk(w, [&](int i, int j, int l, int64_t o) {
        const float kx = __ldg(g.k(0) + i), ky = __ldg(g.k(1) + j), kz = __ldg(g.k(2) + l);
        const float m[3] = {__ldg(g.kz(0) + i), __ldg(g.kz(1) + j), __ldg(g.kz(2) + l)};
        float re = 0.f, im = 0.f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float2 c = C[o + a * w.batch];
            re = fmaf(-m[a], c.y, re);
            im = fmaf(m[a], c.x, im);
        }
        if (S) {
            const float kk[6] = {kx * kx, ky * ky, kz * kz, m[0] * m[1], m[0] * m[2], m[1] * m[2]};
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                const float2 v = S[o + c * w.batch];
                re = fmaf(-kk[c], v.x, re);
                im = fmaf(-kk[c], v.y, im);
            }
        }
        const float mult = l == 0 || 2 * l == g.n2 ? 1.f : 2.f;
        out[i * s0 + j * s1 + l * s2] = solve2(make_float2(re, im), mult * s * inv_k2(kx, ky, kz));
    });
}

int grid_of(const int64_t n[3], const float *tab, LptGrid *g) {
    if (!n) return fail(PMX_ERR_ARG, "null grid_shape");
    for (int a = 0; a < 3; ++a)
        if (n[a] < 1 || n[a] > (1 << 20)) return fail(PMX_ERR_SHAPE, "bad grid shape");
    if (!tab) return fail(PMX_ERR_ARG, "null tables");
    g->n0 = (int)n[0];
    g->n1 = (int)n[1];
    g->n2 = (int)n[2];
    g->n2h = g->n2 / 2 + 1;
    g->tab = tab;
    return PMX_OK;
}

// The walk in the memory order of spectra with the given strides (NULL:
// contiguous) per axis and from one spectrum to the next.
int walk_of(const LptGrid &g, const int64_t *strides, Walk *w) {
    const int n[3] = {g.n0, g.n1, g.n2h};
    const int64_t c[4] = {(int64_t)g.n1 * g.n2h, g.n2h, 1, (int64_t)g.n0 * g.n1 * g.n2h};
    if (!strides) strides = c;
    int ax[3] = {0, 1, 2};
    for (int p = 0; p < 2; ++p)   // largest stride first
        for (int q = 0; q < 2; ++q)
            if (strides[ax[q]] < strides[ax[q + 1]]) {
                const int t = ax[q];
                ax[q] = ax[q + 1];
                ax[q + 1] = t;
            }
    for (int a = 0; a < 3; ++a) {
        if (strides[a] < 1) return fail(PMX_ERR_ARG, "strides must be positive");
        w->ax[a] = ax[a];
        w->n[a] = n[ax[a]];
        w->st[a] = strides[a];
    }
    w->batch = strides[3];
    return PMX_OK;
}

int walk_grid(const Walk &w) {
    const int64_t rows = (int64_t)w.n[0] * w.n[1], need = (rows + LT / 32 - 1) / (LT / 32);
    const int64_t cap = (int64_t)device_sms() * 64;
    return (int)(need < cap ? need : cap);
}
int flat_grid(int64_t n) { return stride_grid(n, LT, 64); }
// one turn per block: a block's stores overlap another one's loads
int disp_grid(int64_t n) {
    return (int)std::min<int64_t>((n + LPT_PB * LT - 1) / (LPT_PB * LT), 1 << 30);
}

int fac_of(const float *fac, int32_t orders, LptFac *f) {
    if (!fac) return fail(PMX_ERR_ARG, "null fac");
    if (orders < 1 || orders > 2) return fail(PMX_ERR_ARG, "orders must be 1 or 2");
    for (int u = 0; u < 4; ++u) f->f[u] = u < 2 * orders ? fac[u] : 0.f;
    f->dev = nullptr;
    return PMX_OK;
}

}  // namespace

extern "C" int pmx_lpt_table_floats(const int64_t grid_shape[3], int64_t *count) {
    LptGrid g;
    float dummy = 0.f;
    int st = grid_of(grid_shape, &dummy, &g);
    if (st) return st;
    if (!count) return fail(PMX_ERR_ARG, "null count");
    *count = table_floats(g.n0, g.n1, g.n2);
    return PMX_OK;
}

extern "C" int pmx_lpt_tables(const int64_t grid_shape[3], const int64_t mesh_shape[3],
                              double ptcl_spacing, double cell_size, float *tables, void *stream) {
    LptGrid g;
    int st = grid_of(grid_shape, tables, &g);
    if (st) return st;
    if (!mesh_shape) return fail(PMX_ERR_ARG, "null mesh_shape");
    if (!(ptcl_spacing > 0) || !(cell_size > 0)) return fail(PMX_ERR_ARG, "sizes must be > 0");
    LptTables t;
    for (int a = 0; a < 3; ++a) {
        t.n[a] = (int)grid_shape[a];
        t.mesh[a] = (int)mesh_shape[a];
        t.unit[a] = cell_size / (double)grid_shape[a];
    }
    const double pi = 3.141592653589793;
    t.period = 2 * pi / ptcl_spacing;
    t.nyq = (float)(pi / ptcl_spacing);
    t.eps = (float)(pi / ptcl_spacing * 1.1920928955078125e-07);
    t.tab = tables;
    k_lpt_tables<<<stride_grid(2 * (g.n0 + g.n1 + g.n2), 128), 128, 0, as_stream(stream)>>>(t);
    PMX_LAUNCH_CHECK("k_lpt_tables");
    return PMX_OK;
}

extern "C" int pmx_lpt_strain(const int64_t grid_shape[3], const float *tables, const float *modes,
                              float scale, float *spec, void *stream) {
    LptGrid g;
    Walk w;
    int st = grid_of(grid_shape, tables, &g);
    if (st || (st = walk_of(g, nullptr, &w))) return st;
    if (!modes || !spec) return fail(PMX_ERR_ARG, "null modes/spec");
    PMX_ALIGNED(8, modes, spec);
    k_lpt_strain<<<walk_grid(w), LT, 0, as_stream(stream)>>>((const float2 *)modes, (float2 *)spec, g,
                                                             w, scale);
    PMX_LAUNCH_CHECK("k_lpt_strain");
    return PMX_OK;
}

extern "C" int pmx_lpt_source(int64_t n, const float *phi, float scale, float *src, void *stream) {
    if (n < 1 || !phi || !src) return fail(PMX_ERR_ARG, "bad lpt source arguments");
    k_lpt_source<1><<<flat_grid(n), LT, 0, as_stream(stream)>>>(phi, src, n, 1, Fields{0, n}, scale);
    PMX_LAUNCH_CHECK("k_lpt_source");
    return PMX_OK;
}

extern "C" int pmx_lpt_grad(const int64_t grid_shape[3], const float *tables, const float *modes,
                            float scale, const float *src2, const int64_t *src2_strides, float *spec,
                            void *stream) {
    LptGrid g;
    Walk w;
    int st = grid_of(grid_shape, tables, &g);
    if (st || (st = walk_of(g, nullptr, &w))) return st;
    if (!modes || !spec || (src2 && !src2_strides)) return fail(PMX_ERR_ARG, "null modes/spec/strides");
    PMX_ALIGNED(8, modes, src2, spec);
    k_lpt_grad<<<walk_grid(w), LT, 0, as_stream(stream)>>>(
        (const float2 *)modes, (const float2 *)src2, src2 ? src2_strides[0] : 0,
        src2 ? src2_strides[1] : 0, src2 ? src2_strides[2] : 0, (float2 *)spec, g, w, scale);
    PMX_LAUNCH_CHECK("k_lpt_grad");
    return PMX_OK;
}

extern "C" int pmx_lpt_disp(const int64_t grid_shape[3], const float *tables, const float *grads,
                            float scale, int32_t orders, const float *fac, const float *fac_dev,
                            int16_t *pmid, float *disp, float *vel, void *stream) {
    LptGrid g;
    LptFac f;
    const float none[4] = {0.f, 0.f, 0.f, 0.f};
    int st = grid_of(grid_shape, tables, &g);
    if (st || (st = fac_of(fac_dev ? none : fac, orders, &f))) return st;
    f.dev = fac_dev;
    if (!grads || !pmid || !disp || !vel) return fail(PMX_ERR_ARG, "null array");
    const int64_t n = (int64_t)g.n0 * g.n1 * g.n2;
    k_lpt_disp<<<disp_grid(n), LT, 0, as_stream(stream)>>>(
        grads, grads + 3 * n, Fields{(int64_t)g.n1 * g.n2, n}, orders, pmid, disp, vel, g, f, scale);
    PMX_LAUNCH_CHECK("k_lpt_disp");
    return PMX_OK;
}

// Parts of pmx_lpt_solve's scratch, in floats: twiddles; three spectra; the half
// rows of up to six fields; six real fields, of which the gradients take the places
// when the strains are used up; the source.
struct SolveScratch {
    MeshGeom g;
    int64_t M, tw, spec, nat, real, src, total;
};
static bool solve_scratch(const LptGrid &g, int32_t orders, SolveScratch *c) {
    if (!mesh_fft_supported(g.n0, g.n1, g.n2)) return false;
    c->g.n0 = g.n0;
    c->g.n1 = g.n1;
    c->g.n2h = g.n2h;
    c->g.nzt = (g.n2h + 3) / 4;
    c->g.unit = (int64_t)g.n0 * g.n1 * 4 * c->g.nzt;
    c->M = (int64_t)g.n0 * g.n1 * g.n2;
    const int64_t nf = orders > 1 ? 6 : 3;
    c->tw = 0;
    c->spec = (2 * mesh_fft_twiddles(g.n0, g.n1, g.n2, nullptr) + 63) / 64 * 64;
    c->nat = c->spec + 2 * (orders > 1 ? 3 : 2) * c->g.unit;
    c->real = c->nat + 2 * nf * c->g.unit;
    c->src = c->real + nf * c->M;
    c->total = c->src + (orders > 1 ? c->M : 0);
    return true;
}

extern "C" int pmx_lpt_solve_floats(const int64_t grid_shape[3], int32_t orders, int64_t *count) {
    LptGrid g;
    float dummy = 0.f;
    int st = grid_of(grid_shape, &dummy, &g);
    if (st) return st;
    if (!count || orders < 1 || orders > 2) return fail(PMX_ERR_ARG, "bad orders or null count");
    SolveScratch c;
    *count = solve_scratch(g, orders, &c) ? c.total : 0;
    return PMX_OK;
}

extern "C" int pmx_lpt_solve(const int64_t grid_shape[3], const float *tables, const float *modes,
                             float scale, int32_t orders, const float *fac, float *scratch,
                             int16_t *pmid, float *disp, float *vel, void *stream) {
    LptGrid g;
    LptFac f;
    SolveScratch c;
    int e = grid_of(grid_shape, tables, &g);
    if (e || (e = fac_of(fac, orders, &f))) return e;
    if (!modes || !scratch || !pmid || !disp || !vel) return fail(PMX_ERR_ARG, "null array");
    PMX_ALIGNED(8, modes);
    PMX_ALIGNED(16, scratch);
    if (!solve_scratch(g, orders, &c)) return fail(PMX_ERR_SHAPE, "no mesh transforms of this shape");
    cudaStream_t st = as_stream(stream);
    if ((e = mesh_rows_prepare(g.n2)) || (e = mesh_cols_prepare(g.n1)) || (e = mesh_xaxis_prepare(g.n0)))
        return e;
    float2 *tx = reinterpret_cast<float2 *>(scratch), *ty = tx + 2 * g.n0, *tz = ty + 2 * g.n1;
    float2 *s0 = reinterpret_cast<float2 *>(scratch + c.spec), *s1 = s0 + c.g.unit;
    float2 *nat = reinterpret_cast<float2 *>(scratch + c.nat);
    float *real = scratch + c.real, *src = scratch + c.src, *g2 = real + 3 * c.M;
    const float2 *md = reinterpret_cast<const float2 *>(modes);
    const int64_t pl = (int64_t)g.n1 * g.n2;
    const float inv = (float)(1.0 / (double)c.M);
    if ((e = mesh_fft_twiddles_dev(g.n0, g.n1, g.n2, tx, st))) return e;
    if (orders > 1) {
        // six strains: X_2, X_1, X_0 are all that the x axis needs to make of them
        if ((e = mesh_xaxis_modes(false, c.g, md, scale, s0, tx, tables, st)) ||
            (e = mesh_cols(MESH_COLS_INV6, 1, c.g, nat, s0, nullptr, ty, tables, st)) ||
            (e = mesh_rows(true, nat, real, tz, 6 * (int64_t)g.n0, g.n1, g.n2, st)))
            return e;
        const int gy = g.n0 < 65535 ? g.n0 : 65535;
        PMX_CUDA(launch_after(k_lpt_source<4>, dim3((unsigned)((pl / 4 + LT - 1) / LT), gy), LT, 0, st,
                              real, src, pl, g.n0, Fields{6 * pl, pl}, inv));
        PMX_LAUNCH_CHECK("k_lpt_source");
        // the gradients of the source's potential: a force with c = 1
        GreenTab gt;
        gt.c[0] = 1.f;
        if ((e = mesh_rows(false, src, nat, tz, g.n0, g.n1, g.n2, st)) ||
            (e = mesh_cols(MESH_COLS_FWD, 1, c.g, nat, s0, s1, ty, tables, st)) ||
            (e = mesh_xaxis(false, 1, c.g, s0, s1, tx, tables, gt, st)) ||
            (e = mesh_cols(MESH_COLS_INV3, 1, c.g, nat, s0, s1, ty, tables, st)) ||
            (e = mesh_rows(true, nat, g2, tz, 3 * (int64_t)g.n0, g.n1, g.n2, st)))
            return e;
    }
    if ((e = mesh_xaxis_modes(true, c.g, md, scale, s0, tx, tables, st)) ||
        (e = mesh_cols(MESH_COLS_INV3, 1, c.g, nat, s0, s1, ty, tables, st)) ||
        (e = mesh_rows(true, nat, real, tz, 3 * (int64_t)g.n0, g.n1, g.n2, st)))
        return e;
    PMX_CUDA(launch_after(k_lpt_disp, disp_grid(c.M), LT, 0, st, real, g2, Fields{3 * pl, pl}, orders,
                          pmid, disp, vel, g, f, inv));
    PMX_LAUNCH_CHECK("k_lpt_disp");
    return PMX_OK;
}

extern "C" int pmx_lpt_disp_adj(int64_t n, const float *disp_cot, const float *vel_cot,
                                int32_t orders, const float *fac, float *grads_cot, void *stream) {
    LptFac f;
    int st = fac_of(fac, orders, &f);
    if (st) return st;
    if (n < 1 || !disp_cot || !vel_cot || !grads_cot) return fail(PMX_ERR_ARG, "null array");
    k_lpt_disp_adj<<<flat_grid(n), LT, 0, as_stream(stream)>>>(disp_cot, vel_cot, orders, grads_cot, n,
                                                               f);
    PMX_LAUNCH_CHECK("k_lpt_disp_adj");
    return PMX_OK;
}

extern "C" int pmx_lpt_src_adj(const int64_t grid_shape[3], const float *tables, const float *spec,
                               const int64_t *strides, float scale, float *src_cot, void *stream) {
    LptGrid g;
    Walk w;
    int st = grid_of(grid_shape, tables, &g);
    if (st || (st = walk_of(g, strides, &w))) return st;
    if (!spec || !src_cot) return fail(PMX_ERR_ARG, "null array");
    PMX_ALIGNED(8, spec, src_cot);
    k_lpt_src_adj<<<walk_grid(w), LT, 0, as_stream(stream)>>>((const float2 *)spec, (float2 *)src_cot,
                                                              g, w, scale);
    PMX_LAUNCH_CHECK("k_lpt_src_adj");
    return PMX_OK;
}

extern "C" int pmx_lpt_source_adj(int64_t n, const float *phi, float scale, const float *src_cot,
                                  float *phi_cot, void *stream) {
    if (n < 1 || !phi || !src_cot || !phi_cot) return fail(PMX_ERR_ARG, "null array");
    k_lpt_source_adj<<<flat_grid(n), LT, 0, as_stream(stream)>>>(phi, src_cot, phi_cot, n, scale);
    PMX_LAUNCH_CHECK("k_lpt_source_adj");
    return PMX_OK;
}

extern "C" int pmx_lpt_modes_adj(const int64_t grid_shape[3], const float *tables,
                                 const float *grads_spec, const float *strain_spec,
                                 const int64_t *strides, float scale, float *modes_cot,
                                 const int64_t *cot_strides, void *stream) {
    LptGrid g;
    Walk w;
    int st = grid_of(grid_shape, tables, &g);
    if (st || (st = walk_of(g, strides, &w))) return st;
    if (!grads_spec || !modes_cot || !cot_strides) return fail(PMX_ERR_ARG, "null array");
    PMX_ALIGNED(8, grads_spec, strain_spec, modes_cot);
    k_lpt_modes_adj<<<walk_grid(w), LT, 0, as_stream(stream)>>>(
        (const float2 *)grads_spec, (const float2 *)strain_spec, (float2 *)modes_cot, cot_strides[0],
        cot_strides[1], cot_strides[2], g, w, scale);
    PMX_LAUNCH_CHECK("k_lpt_modes_adj");
    return PMX_OK;
}
