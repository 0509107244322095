// Internal device/host helpers shared by the libpmx translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string>

#include "../../include/pmx.h"

namespace pmx {

// ---------------------------------------------------------------------------
// error reporting (thread-local message behind pmx_last_error)
// ---------------------------------------------------------------------------
void set_error(const std::string &msg);
void clear_error();
int fail(int code, const std::string &msg);
int cuda_status(cudaError_t e, const char *what);

#define PMX_CUDA(call)                                                        \
    do {                                                                      \
        cudaError_t e_ = (call);                                              \
        if (e_ != cudaSuccess) return ::pmx::cuda_status(e_, #call);          \
    } while (0)

#define PMX_LAUNCH_CHECK(what)                                                \
    do {                                                                      \
        cudaError_t e_ = cudaGetLastError();                                  \
        if (e_ != cudaSuccess) return ::pmx::cuda_status(e_, what);           \
    } while (0)

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

int device_sms();

// Grid for grid-stride kernels: enough blocks to fill every SM several times,
// never more than the work needs.
inline int stride_grid(int64_t work, int threads, int per_sm = 8) {
    int64_t need = (work + threads - 1) / threads;
    int64_t cap = (int64_t)device_sms() * per_sm;
    if (need < 1) need = 1;
    return (int)(need < cap ? need : cap);
}

// ---------------------------------------------------------------------------
// enmesh parameters (pm_util.py:33-156), resolved on the host from
// pmx_enmesh_spec.  The kernels always work on 3 internal axes; a dim < 3
// problem is embedded as singleton leading axes (pmid 0, disp 0, shape 1),
// which reproduces the reference's fractions exactly (the padded factors
// are 1 and 0).
// ---------------------------------------------------------------------------
struct EmParams {
    int dim;           // user spatial dims
    int pad;           // 3 - dim: internal axes [0, pad) are singleton
    int wrap[3];       // s1 per internal axis (0: no wrapping, s1 = None)
    int drop;          // without wrapping: negative indices -> s2
    int64_t shape[3];  // s2 per internal axis
    int64_t stride[3]; // mesh cell stride per internal axis
    int f64;           // 1: non-default (float64) branch, pm_util.py:99-118
    // default branch (pm_util.py:119-137)
    float cellf;       // a1 as float32
    float cell_inv;    // exact_inverse(cellf)
    int i12[3];        // integer part of offset / a1 (jnp.divmod)
    float d12[3];      // remainder, cast to float32
    // float64 branch
    double a1d, a2d;
    double b12[3];
    double L[3];       // s1 * a1
    float a2f;
    // scatter/gather adjoints divide disp_cot by this (f32 of cell_size or
    // conf.cell_size), scatter.py:116 / gather.py:110
    float cot_div;
};

// Whether every pointer is on `bytes` bytes (NULL is): what kernels that read pairs or
// 16 bytes at a time need of the caller's arrays.
template <class... P>
bool aligned(size_t bytes, const P *...p) {
    return ((reinterpret_cast<uintptr_t>(p) % bytes == 0) && ...);
}

int make_em_params(const pmx_enmesh_spec *spec, EmParams *p);
// 1 / y if y is a power of two well inside the float range, else 0.
float exact_inverse(float y);

// 3-D mesh transforms of the Poisson solve by this library's own kernels
// (pmx_mesh_fft.cuh; pmx_mesh_rows.cu, pmx_mesh_cols.cu, pmx_mesh_x.cu).
struct MeshGeom {
    int64_t n0, n1;      // planes and rows
    int nzt;             // blocks of 4 kz values: ceil((n2 / 2 + 1) / 4)
    int n2h;
    int64_t unit;        // complex values of one spectrum: n0 n1 4 nzt
};

constexpr int MESH_SLOTS = 16;
struct GreenTab {
    float c[MESH_SLOTS];   // 1.5 Omega_m / N of each slot
};
bool mesh_fft_supported(int64_t n0, int64_t n1, int64_t n2);
// Writes the twiddle tables to t (unless NULL); returns their length.
int64_t mesh_fft_twiddles(int64_t n0, int64_t n1, int64_t n2, float2 *t);
// The same tables computed on the device (t in device memory).
int mesh_fft_twiddles_dev(int64_t n0, int64_t n1, int64_t n2, float2 *t, cudaStream_t st);
// x axis of contiguous modes (n0, n1, n2h), p = scale modes / k^2: spectra X_2, X_1,
// X_0 (grads false: inverse transforms of kx^2 p, kx p, p) or G_0, Q (grads true: of
// i kx p, -p), one after the other.
int mesh_xaxis_modes(bool grads, const MeshGeom &g, const float2 *modes, float scale, float2 *spec,
                     const float2 *tw, const float *kt, cudaStream_t st);
int mesh_rows_prepare(int64_t n2);   // once per workspace: shared-memory opt-ins
int mesh_rows_factors(int64_t n2, int *R1, int *R2);   // of the half length
int mesh_cols_prepare(int64_t n1);
int mesh_xaxis_prepare(int64_t n0);
// z axis of `planes` consecutive planes: real <-> nat.
int mesh_rows(bool inv, const void *in, void *out, const float2 *tw, int64_t planes, int64_t n1,
              int64_t n2, cudaStream_t st);
enum { MESH_COLS_FWD, MESH_COLS_ADJ, MESH_COLS_INV1, MESH_COLS_INV3, MESH_COLS_INV6 };
// y axis of nslot slots: nat <-> spectra (one, or two: spec0 and spec1).
int mesh_cols(int kind, int nslot, const MeshGeom &g, float2 *nat, float2 *spec0, float2 *spec1,
              const float2 *tw, const float *kt, cudaStream_t st);
// Both axes of n1 x n1 planes (FWD, INV1, INV3): real planes <-> spectra.  FWD leaves
// the planes filled with -1, as the next density deposit wants them.
// prepare: once per workspace; *fits: whether there are kernels for these planes.
int mesh_plane_prepare(int64_t n1, int64_t n2, bool *fits);
int mesh_plane(int kind, int nslot, const MeshGeom &g, float *mesh, float2 *spec0, float2 *spec1,
               const float2 *twy, const float2 *twz, const float *kt, cudaStream_t st);
int mesh_xaxis(bool adj, int nslot, const MeshGeom &g, float2 *s0, float2 *s1, const float2 *tw,
               const float *kt, const GreenTab &gt, cudaStream_t st);

// Fused x-axis pass of the Poisson solve (pmx_fft.cu).  Forward (adj =
// false): in = FFT_yz(rho) (n0, n1, n2h), out = the three gradient spectra
// (n0, 3, n1, n2h) after the inverse x transform.  Adjoint: in = FFT_yz of
// the three mesh cotangents (n0, 3, n1, n2h), out = (n0, n1, n2h).
// Complex rows hold n2h values at a stride of rs >= n2h elements.
bool xpass_supported(int64_t n0);
int xpass(bool adj, const float2 *in, float2 *out, const float *kt, const float2 *tw, int64_t n0,
          int64_t n1, int64_t n2h, int64_t rs, float c, cudaStream_t st);
// n2h rounded up to a multiple of 4 complex values (32 bytes): the complex
// row stride of the plane-kernel path, so every column tile of a plane
// covers whole 32-byte sectors (HBM3e has no byte-masked writes).
inline int64_t padded_row(int64_t n2h) { return (n2h + 3) & ~(int64_t)3; }
void xpass_twiddles(int64_t n, float2 *host);

// 2-D (y, z) transforms of consecutive planes (pmx_fft.cu): forward real
// (n1, n2) -> complex (n1, n2/2+1) at row stride padded_row(n2/2+1); inverse
// complex -> real through a scratch plane per cluster (n1 * padded_row
// complex values each, plane_max_clusters of them).  One thread-block cluster
// per plane.  ptw holds plane_twiddles(n1, n2) (2 n1 + 1 entries).
bool plane_supported(int64_t n1, int64_t n2);
// c16: clusters of 16 CTAs (non-portable size) instead of 8.
int plane_max_clusters(int64_t n1, int64_t n2, bool c16, int *ncl);
int plane_fft(bool inv, const void *in, void *out, const float2 *ptw, int64_t nplanes, int64_t n1,
              int64_t n2, float2 *scratch, int max_clusters, bool c16, cudaStream_t st);
void plane_twiddles(int64_t n1, int64_t n2, float2 *host);

__device__ __forceinline__ int pymod(int x, int m) {
    int r = x % m;
    return r < 0 ? r + m : r;
}

// i modulo n; positions within one period of the box, the usual ones, take an
// addition instead of an integer division.
__device__ __forceinline__ int fast_mod(int i, int n) {
    if ((unsigned)i < (unsigned)n) return i;
    i += i < 0 ? n : -n;
    return (unsigned)i < (unsigned)n ? i : pymod(i, n);
}

// x / y as IEEE division gives it, by multiplying with inv = 1 / y where that
// is exact (y a power of two; inv = 0 otherwise).
__device__ __forceinline__ float div_or_mul(float x, float y, float inv) {
    return inv != 0.f ? __fmul_rn(x, inv) : __fdiv_rn(x, y);
}

__device__ __forceinline__ float sgnf(float x) {
    // jnp.sign: -1, 0 (signed), +1
    return x > 0.f ? 1.f : (x < 0.f ? -1.f : x);
}

// jnp.remainder for doubles (sign of divisor).  Within one period either way
// fmod is x or, exactly, x - m; its general loop is what costs at this device's
// float64 rate.
__device__ __forceinline__ double pyfmod(double x, double m) {
    if (x >= 0.0 && x < m) return x;
    if (x >= m && x < 2.0 * m) return __dsub_rn(x, m);
    double t = fmod(x, m);
    if (t != 0.0 && ((t < 0.0) != (m < 0.0))) t = __dadd_rn(t, m);
    return t;
}

// jnp.floor_divide for doubles (CPython float_divmod + round half away)
__device__ __forceinline__ double floordiv(double x, double y) {
    if (x >= 0.0 && y > 0.0 && x < 1e9 * y) {
        // the quotient's floor, corrected by its remainder, which is exact in
        // one fused operation: what fmod and the division below come to
        double q = floor(__ddiv_rn(x, y));
        const double r = fma(-q, y, x);
        if (r < 0.0) q -= 1.0;
        else if (r >= y) q += 1.0;
        return q;
    }
    double mod = fmod(x, y);
    double div = __ddiv_rn(__dsub_rn(x, mod), y);
    if (mod != 0.0 && ((y < 0.0) != (mod < 0.0))) div = __dsub_rn(div, 1.0);
    return round(div);
}

// Per-axis neighbour data: indices (wrapped by s1, not dropped), fractions
// and the signs sign(-d2) used by the fraction gradients.
struct Axis {
    int i[2];
    float w[2];
    float s[2];
    int u;  // unwrapped index of the lower neighbour (hot path only)
};

__device__ __forceinline__ void enmesh_axis(const EmParams &p, int a, int pm, float d,
                                            Axis &ax) {
    if (a < p.pad) {
        ax.i[0] = 0; ax.i[1] = 0;
        ax.w[0] = 1.f; ax.w[1] = 0.f;
        ax.s[0] = 0.f; ax.s[1] = 1.f;
        return;
    }
    if (!p.f64) {
        int ip = pm - p.i12[a];
        float x = div_or_mul(__fsub_rn(d, p.d12[a]), p.cellf, p.cell_inv);
        int fl = (int)floorf(x);
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
            int ii = fl + nb;
            float d2 = __fsub_rn(x, (float)ii);
            ax.w[nb] = __fsub_rn(1.f, fabsf(d2));
            ax.s[nb] = sgnf(-d2);
            // without wrapping, the reference's int16 sum (two's complement)
            ax.i[nb] = p.wrap[a] ? fast_mod(ii + ip, p.wrap[a]) : (int)(short)(ii + ip);
        }
    } else {
        double P = __dsub_rn(__dadd_rn(__dmul_rn((double)pm, p.a1d), (double)d), p.b12[a]);
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
            double x = nb ? __dadd_rn(P, p.a2d) : P;
            if (p.wrap[a]) x = pyfmod(x, p.L[a]);
            double q = floordiv(x, p.a2d);
            double d2 = __dsub_rn(P, __dmul_rn(q, p.a2d));
            if (p.wrap[a] && fabs(d2) >= 0.25 * p.L[a])   // below, the rounded quotient is 0
                d2 = __dsub_rn(d2, __dmul_rn(rint(__ddiv_rn(d2, p.L[a])), p.L[a]));
            float d2f = __fdiv_rn((float)d2, p.a2f);
            ax.w[nb] = __fsub_rn(1.f, fabsf(d2f));
            ax.s[nb] = sgnf(-d2f);
            ax.i[nb] = (int)(short)(int)q;
        }
    }
    // pm_util.py:139-140: without wrapping, negative indices are set to s2
    if (!p.wrap[a] && p.drop) {
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
            if (ax.i[nb] < 0) ax.i[nb] = (int)p.shape[a];
    }
}

// Loads one particle (3 internal axes) from row-major (n, dim) arrays.
template <typename IT>
__device__ __forceinline__ void load_particle(const EmParams &p, const IT *pmid,
                                              const float *disp, int64_t q,
                                              int pm[3], float dd[3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int u = a - p.pad;
        if (u >= 0) {
            pm[a] = (int)pmid[q * p.dim + u];
            dd[a] = disp[q * p.dim + u];
        } else {
            pm[a] = 0;
            dd[a] = 0.f;
        }
    }
}

// Raveled cell of neighbour k (bit a of k selects neighbour along internal
// axis a, matching pm_util.py:95-97), or -1 when dropped (index >= s2).
__device__ __forceinline__ int64_t cell_of(const EmParams &p, const Axis ax[3], int k) {
    int64_t off = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int ii = ax[a].i[(k >> a) & 1];
        // wrapped indices are never negative; a negative one can only come
        // from int16 overflow of a huge displacement and is dropped
        if (ii < 0 || (int64_t)ii >= p.shape[a]) return -1;
        off += (int64_t)ii * p.stride[a];
    }
    return off;
}

__device__ __forceinline__ float frac_of(const Axis ax[3], int k) {
    return __fmul_rn(__fmul_rn(ax[0].w[k & 1], ax[1].w[(k >> 1) & 1]), ax[2].w[(k >> 2) & 1]);
}

// d frac / d (x_a / cell): sign(-d2_a) times the product of the other axes'
// fractions in the reference's order (a+1, ..., dim-1, 0, ..., a-1).
__device__ __forceinline__ void frac_grad_of(const Axis ax[3], int k, float g[3]) {
    float w0 = ax[0].w[k & 1], w1 = ax[1].w[(k >> 1) & 1], w2 = ax[2].w[(k >> 2) & 1];
    g[0] = __fmul_rn(ax[0].s[k & 1], __fmul_rn(w1, w2));
    g[1] = __fmul_rn(ax[1].s[(k >> 1) & 1], __fmul_rn(w2, w0));
    g[2] = __fmul_rn(ax[2].s[(k >> 2) & 1], __fmul_rn(w0, w1));
}

// (double)x: the exponent rebiased and the mantissa shifted by integer
// operations for normal numbers.  The float64 unit, which also converts, runs
// at about two operations per clock and SM here: dot products of six
// conversions and four operations held up the kick/drift adjoint passes (256^3
// particles on 256^3: 0.68 against 0.63 ms with three operations and no
// conversion).
__device__ __forceinline__ double to_f64(float x) {
    const unsigned u = __float_as_uint(x), e = u & 0x7f800000u;
    if (e == 0u || e == 0x7f800000u) return (double)x;   // zero, subnormal, inf, NaN
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)),
                            (int)(u << 29));
}

// Programmatic dependent launch: a kernel launched by launch_after is set up while
// the stream's previous kernel ends; it waits in after_previous() until that one is
// done and its memory operations are visible, before it touches global memory.
// Every kernel of such a chain waits, so each sees all earlier ones.  It saves the
// 1 to 2 us between two kernels.  Without such a launch after_previous() returns at
// once.  The next kernel is set up as blocks exit: allowed from a block's start on
// (griddepcontrol.launch_dependents), its waiting blocks take the room of the large
// meshes' kernels (8 steps of 256^3 particles on 512^3: 57.9 ms against 28.5).
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class... K, class... A>
cudaError_t launch_after(void (*fn)(K...), dim3 grid, int block, size_t smem, cudaStream_t st,
                         A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, K(args)...);
}

// Deterministic block sum of one double per thread; thread 0 gets the total.
template <int THREADS>
__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 0; w < THREADS / 32; ++w) t += sh[w];
    }
    __syncthreads();
    return t;
}

}  // namespace pmx
