// Generic CIC mesh operators: enmesh, scatter, gather and their VJPs.
//
// These back the general pmwd signatures (any dim 1..3, channels, offset,
// non-default cell size): pmwd/scatter.py:8-150, pmwd/gather.py:8-144,
// pmwd/particles.py:212-254.  The Poisson-force hot path uses the fused,
// specialised kernels in pmx_force.cu.
//
// One thread per particle.  Scatter-type updates use float32 global reductions
// (red.global.add through atomicAdd with the result unused), like the
// reference's XLA scatter-add.
//
// Two sets of kernels.  The default enmesh in 3-D with one or three channels
// (k_*_cic: any periodic particle set on its own mesh, the usual call) has
// every neighbour in the mesh, so rows are addressed by 32-bit offsets within
// an x-plane, both z neighbours are read together and reductions of adjacent
// cells are merged.  The general kernels cover everything else: other cell
// sizes (the float64 branch), other dimensions, dropped neighbours, any number
// of channels.  What bounds the k_*_cic kernels is the L2's reductions and, for
// clustered sets, its reads.  With the general kernels / with these: scatter and
// its VJP, 256^3 clustered particles on 256^3, 1.56 / 0.83 ms; gather of three
// channels and its VJP, 175 x 125 x 225, 0.90 / 0.50 ms.

#include <cmath>
#include <cstdio>
#include <mutex>
#include <string>

#include "pmx_internal.cuh"

namespace pmx {

static thread_local std::string g_err;

void set_error(const std::string &msg) { g_err = msg; }
void clear_error() { g_err.clear(); }
int fail(int code, const std::string &msg) {
    g_err = msg;
    return code;
}
int cuda_status(cudaError_t e, const char *what) {
    g_err = std::string(what) + ": " + cudaGetErrorString(e);
    return PMX_ERR_CUDA;
}

int device_sms() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
    if (cached[dev] == 0) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
            v = 152;
        cached[dev] = v;
    }
    return cached[dev];
}

// jnp.divmod(b12, a1) for floats, done once on the host (pm_util.py:120).
static void host_float_divmod(double x, double y, double *div, double *mod) {
    double m = std::fmod(x, y);
    double d = (x - m) / y;
    if (m != 0.0 && ((y < 0.0) != (m < 0.0))) {
        m += y;
        d -= 1.0;
    }
    *div = std::round(d);  // half away from zero, like lax.round
    *mod = m;
}

float exact_inverse(float y) {
    int e = 0;
    return std::frexp(y, &e) == 0.5f && e > -126 && e < 126 ? 1.f / y : 0.f;
}

int make_em_params(const pmx_enmesh_spec *s, EmParams *p) {
    if (!s) return fail(PMX_ERR_ARG, "null enmesh spec");
    if (s->dim < 1 || s->dim > 3) return fail(PMX_ERR_ARG, "dim must be 1, 2 or 3");
    if (!(s->conf_cell_size > 0)) return fail(PMX_ERR_ARG, "conf_cell_size must be > 0");
    p->dim = s->dim;
    p->pad = 3 - s->dim;
    // all wrap_shape entries 0: no periodic wrapping (s1 = None)
    bool nowrap = true;
    for (int u = 0; u < s->dim; ++u) nowrap = nowrap && s->wrap_shape[u] == 0;
    p->drop = nowrap && s->drop;
    for (int a = 0; a < 3; ++a) {
        int u = a - p->pad;
        if (u < 0) {
            p->wrap[a] = 1;
            p->shape[a] = 1;
        } else if (nowrap) {
            if (s->mesh_shape[u] <= 0) return fail(PMX_ERR_ARG, "mesh_shape must be > 0");
            p->wrap[a] = 0;
            p->shape[a] = s->mesh_shape[u];
        } else {
            if (s->wrap_shape[u] <= 0) return fail(PMX_ERR_ARG, "wrap_shape must be > 0 (or all 0)");
            if (s->mesh_shape[u] <= 0) return fail(PMX_ERR_ARG, "mesh_shape must be > 0");
            p->wrap[a] = s->wrap_shape[u];
            p->shape[a] = s->mesh_shape[u];
        }
    }
    p->stride[2] = 1;
    p->stride[1] = p->shape[2];
    p->stride[0] = p->shape[1] * p->shape[2];
    p->f64 = s->cell_size > 0 ? 1 : 0;
    p->cellf = (float)s->conf_cell_size;
    p->cell_inv = exact_inverse(p->cellf);
    p->a1d = s->conf_cell_size;
    p->a2d = s->cell_size > 0 ? s->cell_size : s->conf_cell_size;
    p->a2f = (float)p->a2d;
    for (int a = 0; a < 3; ++a) {
        int u = a - p->pad;
        double off = u >= 0 ? s->offset[u] : 0.0;
        double div, mod;
        host_float_divmod(off, (double)p->cellf, &div, &mod);
        p->i12[a] = (int)(int16_t)(int64_t)div;
        p->d12[a] = (float)mod;
        p->b12[a] = off;
        p->L[a] = (double)p->wrap[a] * p->a1d;
    }
    p->cot_div = (float)(s->cell_size > 0 ? s->cell_size : s->conf_cell_size);
    return PMX_OK;
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------

__global__ void k_enmesh(EmParams p, const int16_t *__restrict__ pmid,
                         const float *__restrict__ disp, int64_t n, int32_t *ind,
                         float *frac, float *frac_grad) {
    const int nk = 1 << p.dim;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        int pm[3];
        float dd[3];
        load_particle(p, pmid, disp, q, pm, dd);
        Axis ax[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) enmesh_axis(p, a, pm[a], dd[a], ax[a]);
        for (int ku = 0; ku < nk; ++ku) {
            int k = ku << p.pad;  // user neighbour bits -> internal bits
            frac[q * nk + ku] = frac_of(ax, k);
            if (ind) {
                for (int u = 0; u < p.dim; ++u) {
                    int a = u + p.pad;
                    ind[(q * nk + ku) * p.dim + u] = ax[a].i[(k >> a) & 1];
                }
            }
            if (frac_grad) {
                float g[3];
                frac_grad_of(ax, k, g);
                for (int u = 0; u < p.dim; ++u)
                    frac_grad[(q * nk + ku) * p.dim + u] = g[u + p.pad];
            }
        }
    }
}

__global__ void k_scatter(EmParams p, const int16_t *__restrict__ pmid,
                          const float *__restrict__ disp, int64_t n,
                          const float *__restrict__ val, float val_scalar, int64_t chan,
                          float *mesh) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        int pm[3];
        float dd[3];
        load_particle(p, pmid, disp, q, pm, dd);
        Axis ax[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) enmesh_axis(p, a, pm[a], dd[a], ax[a]);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            int64_t cell = cell_of(p, ax, k);
            if (cell < 0) continue;
            float f = frac_of(ax, k);
            if (val) {
                for (int64_t c = 0; c < chan; ++c)
                    atomicAdd(mesh + cell * chan + c, __fmul_rn(val[q * chan + c], f));
            } else {
                atomicAdd(mesh + cell, __fmul_rn(val_scalar, f));
            }
        }
    }
}

__global__ void k_scatter_adj(EmParams p, const int16_t *__restrict__ pmid,
                              const float *__restrict__ disp, int64_t n,
                              const float *__restrict__ val, float val_scalar, int64_t chan,
                              const float *__restrict__ mesh_cot, float *disp_cot,
                              float *val_cot) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        int pm[3];
        float dd[3];
        load_particle(p, pmid, disp, q, pm, dd);
        Axis ax[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) enmesh_axis(p, a, pm[a], dd[a], ax[a]);
        float dc[3] = {0.f, 0.f, 0.f};
        for (int k = 0; k < 8; ++k) {
            int64_t cell = cell_of(p, ax, k);
            float g[3];
            frac_grad_of(ax, k, g);
            float f = frac_of(ax, k);
            float s = 0.f;
            for (int64_t c = 0; c < chan; ++c) {
                float m = cell >= 0 ? mesh_cot[cell * chan + c] : 0.f;
                float v = val ? val[q * chan + c] : val_scalar;
                s = __fadd_rn(s, __fmul_rn(m, v));
                if (val_cot) {
                    float *o = val_cot + q * chan + c;
                    float prev = k == 0 ? 0.f : *o;
                    *o = __fadd_rn(prev, __fmul_rn(m, f));
                }
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) dc[a] = __fadd_rn(dc[a], __fmul_rn(s, g[a]));
        }
        for (int u = 0; u < p.dim; ++u)
            disp_cot[q * p.dim + u] = __fdiv_rn(dc[u + p.pad], p.cot_div);
    }
}

__global__ void k_gather(EmParams p, const int16_t *__restrict__ pmid,
                         const float *__restrict__ disp, int64_t n,
                         const float *__restrict__ mesh, int64_t chan,
                         const float *__restrict__ val, float val_scalar, float *out) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        int pm[3];
        float dd[3];
        load_particle(p, pmid, disp, q, pm, dd);
        Axis ax[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) enmesh_axis(p, a, pm[a], dd[a], ax[a]);
        int64_t cells[8];
        float fr[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            cells[k] = cell_of(p, ax, k);
            fr[k] = frac_of(ax, k);
        }
        for (int64_t c = 0; c < chan; ++c) {
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                float m = cells[k] >= 0 ? mesh[cells[k] * chan + c] : 0.f;
                s = __fadd_rn(s, __fmul_rn(m, fr[k]));
            }
            float v = val ? val[q * chan + c] : val_scalar;
            out[q * chan + c] = __fadd_rn(v, s);
        }
    }
}

__global__ void k_gather_adj(EmParams p, const int16_t *__restrict__ pmid,
                             const float *__restrict__ disp, int64_t n,
                             const float *__restrict__ mesh, int64_t chan,
                             const float *__restrict__ val_cot, float *disp_cot,
                             float *mesh_cot) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        int pm[3];
        float dd[3];
        load_particle(p, pmid, disp, q, pm, dd);
        Axis ax[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) enmesh_axis(p, a, pm[a], dd[a], ax[a]);
        float dc[3] = {0.f, 0.f, 0.f};
        for (int k = 0; k < 8; ++k) {
            int64_t cell = cell_of(p, ax, k);
            float g[3];
            frac_grad_of(ax, k, g);
            float f = frac_of(ax, k);
            float s = 0.f;
            for (int64_t c = 0; c < chan; ++c) {
                float vc = val_cot[q * chan + c];
                float m = cell >= 0 ? mesh[cell * chan + c] : 0.f;
                s = __fadd_rn(s, __fmul_rn(vc, m));
                if (cell >= 0) atomicAdd(mesh_cot + cell * chan + c, __fmul_rn(vc, f));
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) dc[a] = __fadd_rn(dc[a], __fmul_rn(s, g[a]));
        }
        for (int u = 0; u < p.dim; ++u)
            disp_cot[q * p.dim + u] = __fdiv_rn(dc[u + p.pad], p.cot_div);
    }
}

// --------------------------------------------------------------------------
// default enmesh, 3-D, NC = 1 or 3 channels
// --------------------------------------------------------------------------

struct Cic {
    int wrap[3], i12[3];
    float d12[3], cell, inv, div, div_inv;
    int64_t s0;      // cells of an x-plane of the mesh array
    unsigned s1;     // cells of a row
    bool join;       // about one cell per particle: hand values to the next lane
    bool pair;       // the added-to array starts on 8 bytes
};

struct CicAxis {
    int i[2];
    float w[2], s[2];
};

__device__ __forceinline__ void cic_axes(const Cic &p, const int16_t *__restrict__ pmid,
                                         const float *__restrict__ disp, int64_t q, CicAxis ax[3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float x = div_or_mul(__fsub_rn(disp[3 * q + a], p.d12[a]), p.cell, p.inv);
        const int fl = (int)floorf(x);
        const float d0 = __fsub_rn(x, (float)fl), d1 = __fsub_rn(x, (float)(fl + 1));
        ax[a].w[0] = __fsub_rn(1.f, fabsf(d0));
        ax[a].w[1] = __fsub_rn(1.f, fabsf(d1));
        ax[a].s[0] = sgnf(-d0);
        ax[a].s[1] = sgnf(-d1);
        ax[a].i[0] = fast_mod(fl + (int)pmid[3 * q + a] - p.i12[a], p.wrap[a]);
        ax[a].i[1] = ax[a].i[0] + 1 == p.wrap[a] ? 0 : ax[a].i[0] + 1;
    }
}

// Row r (bit 0: x neighbour, bit 1: y neighbour): its cells' offset from the
// start of the array is x * s0 + the 32-bit offset.
__device__ __forceinline__ int64_t cic_plane(const Cic &p, const CicAxis ax[3], int r) {
    return ax[0].i[r & 1] * p.s0;
}
__device__ __forceinline__ unsigned cic_row(const Cic &p, const CicAxis ax[3], int r) {
    return (unsigned)ax[1].i[r >> 1] * p.s1;
}

// The NC channels at both z neighbours of a row, m[bit][c].
template <int NC>
__device__ __forceinline__ void cic_read(const Cic &p, const CicAxis ax[3], int r,
                                         const float *__restrict__ mesh, float (&m)[2][NC]) {
    const float *b = mesh + cic_plane(p, ax, r) * NC;
    const unsigned y = cic_row(p, ax, r);
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
        for (int c = 0; c < NC; ++c) m[z][c] = __ldg(b + ((y + (unsigned)ax[2].i[z]) * NC + c));
}

// Adds v[c] (w_x w_y) w_z to the eight neighbours (every lane of a warp calls
// it).  Two ways to merge reductions, chosen per warp:
// join: a lane hands its upper z neighbours' values to the next lane if that
// one's lower cells are the same, the rule among neighbours on the lattice at
// one cell per particle.  Taken where at least 12 of 32 lanes can.
// pair (arrays on 8 bytes): adjacent floats of the row at an even offset take
// one 8-byte reduction: finer meshes and particles that have left the lattice.
template <int NC>
__device__ __forceinline__ void cic_add(const Cic &p, bool act, const CicAxis ax[3],
                                        const float (&v)[NC], float *mesh) {
    const int i0 = ax[2].i[0], i1 = ax[2].i[1];
    bool join = false, next = false, joined = false;
    if (p.join) {
        const int lane = threadIdx.x & 31;
        const unsigned o = act ? cic_row(p, ax, 0) + (unsigned)i0 : 0u;
        const int x = act ? ax[0].i[0] : -1;
        const unsigned po = __shfl_up_sync(0xffffffffu, o, 1);
        const int px = __shfl_up_sync(0xffffffffu, x, 1);
        join = act && lane > 0 && px == x && po + 1 == o && i0 != 0;
        const unsigned jm = __ballot_sync(0xffffffffu, join);
        joined = __popc(jm) >= 12;
        next = (jm >> lane >> 1) & 1;
    }
    if (joined) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float fxy = __fmul_rn(ax[0].w[r & 1], ax[1].w[r >> 1]);
            const float fa = __fmul_rn(fxy, ax[2].w[0]), fb = __fmul_rn(fxy, ax[2].w[1]);
            float *b = mesh + cic_plane(p, ax, r) * NC;
            const unsigned y = cic_row(p, ax, r);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                float e = __fmul_rn(v[c], fa);
                const float u = __fmul_rn(v[c], fb), pu = __shfl_up_sync(0xffffffffu, u, 1);
                if (join) e += pu;
                if (act) {
                    atomicAdd(b + ((y + (unsigned)i0) * NC + c), e);
                    if (!next) atomicAdd(b + ((y + (unsigned)i1) * NC + c), u);
                }
            }
        }
        return;
    }
    if (!act) return;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float fxy = __fmul_rn(ax[0].w[r & 1], ax[1].w[r >> 1]);
        const float fa = __fmul_rn(fxy, ax[2].w[0]), fb = __fmul_rn(fxy, ax[2].w[1]);
        const int64_t plane = cic_plane(p, ax, r) * NC;
        float *b = mesh + plane, e[2 * NC];
        const unsigned y = cic_row(p, ax, r);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            e[c] = __fmul_rn(v[c], fa);
            e[NC + c] = __fmul_rn(v[c], fb);
        }
        const unsigned o0 = (y + (unsigned)i0) * NC, o1 = (y + (unsigned)i1) * NC;
        if (!p.pair || i1 != i0 + 1) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                atomicAdd(b + (o0 + c), e[c]);
                atomicAdd(b + (o1 + c), e[NC + c]);
            }
        } else if (((o0 + (unsigned)plane) & 1u) == 0) {   // 2 NC floats in NC pairs
#pragma unroll
            for (int c = 0; c < NC; ++c)
                atomicAdd(reinterpret_cast<float2 *>(b + (o0 + 2 * c)),
                          make_float2(e[2 * c], e[2 * c + 1]));
        } else {                                           // a single one at either end
            atomicAdd(b + o0, e[0]);
#pragma unroll
            for (int c = 0; c + 1 < NC; ++c)
                atomicAdd(reinterpret_cast<float2 *>(b + (o0 + 2 * c + 1)),
                          make_float2(e[2 * c + 1], e[2 * c + 2]));
            atomicAdd(b + (o0 + 2 * NC - 1), e[2 * NC - 1]);
        }
    }
}

template <int NC>
__device__ __forceinline__ void ld_val(const float *__restrict__ val, float scalar, int64_t q,
                                       float (&v)[NC]) {
#pragma unroll
    for (int c = 0; c < NC; ++c) v[c] = val ? val[q * NC + c] : scalar;
}

template <int NC>
__global__ void __launch_bounds__(256) k_scatter_cic(Cic p, const int16_t *__restrict__ pmid,
                                                     const float *__restrict__ disp, int64_t n,
                                                     const float *__restrict__ val,
                                                     float val_scalar, float *mesh) {
    for (int64_t q0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); q0 < n;
         q0 += (int64_t)gridDim.x * blockDim.x) {   // warp-uniform
        const int64_t q = q0 + (threadIdx.x & 31);
        CicAxis ax[3] = {};
        float v[NC] = {};
        if (q < n) {
            cic_axes(p, pmid, disp, q, ax);
            ld_val<NC>(val, val_scalar, q, v);
        }
        cic_add<NC>(p, q < n, ax, v, mesh);
    }
}

// Position term sum_k t_k dfrac_k / cell of a row's two values t[bit].
__device__ __forceinline__ void cic_grad(const CicAxis ax[3], int r, const float t[2], float c[3]) {
    const int bx = r & 1, by = r >> 1;
    const float T = fmaf(t[1], ax[2].w[1], t[0] * ax[2].w[0]);
    const float D = fmaf(t[1], ax[2].s[1], t[0] * ax[2].s[0]);
    c[0] = fmaf(ax[0].s[bx] * ax[1].w[by], T, c[0]);
    c[1] = fmaf(ax[0].w[bx] * ax[1].s[by], T, c[1]);
    c[2] = fmaf(ax[0].w[bx] * ax[1].w[by], D, c[2]);
}

template <int NC>
__global__ void __launch_bounds__(256) k_scatter_adj_cic(
    Cic p, const int16_t *__restrict__ pmid, const float *__restrict__ disp, int64_t n,
    const float *__restrict__ val, float val_scalar, const float *__restrict__ mesh_cot,
    float *disp_cot, float *val_cot) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        CicAxis ax[3];
        float v[NC], g[NC] = {}, c[3] = {0.f, 0.f, 0.f};
        cic_axes(p, pmid, disp, q, ax);
        ld_val<NC>(val, val_scalar, q, v);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float m[2][NC], t[2] = {0.f, 0.f};
            cic_read<NC>(p, ax, r, mesh_cot, m);
            const float f = ax[0].w[r & 1] * ax[1].w[r >> 1];
#pragma unroll
            for (int k = 0; k < NC; ++k) {
                t[0] = fmaf(m[0][k], v[k], t[0]);
                t[1] = fmaf(m[1][k], v[k], t[1]);
                g[k] = fmaf(f, fmaf(m[1][k], ax[2].w[1], m[0][k] * ax[2].w[0]), g[k]);
            }
            cic_grad(ax, r, t, c);
        }
        if (val_cot) {
#pragma unroll
            for (int k = 0; k < NC; ++k) val_cot[q * NC + k] = g[k];
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) disp_cot[3 * q + a] = div_or_mul(c[a], p.div, p.div_inv);
    }
}

template <int NC>
__global__ void __launch_bounds__(256) k_gather_cic(Cic p, const int16_t *__restrict__ pmid,
                                                    const float *__restrict__ disp, int64_t n,
                                                    const float *__restrict__ mesh,
                                                    const float *__restrict__ val,
                                                    float val_scalar, float *out) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        CicAxis ax[3];
        float v[NC], g[NC] = {};
        cic_axes(p, pmid, disp, q, ax);
        ld_val<NC>(val, val_scalar, q, v);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float m[2][NC];
            cic_read<NC>(p, ax, r, mesh, m);
            const float f = ax[0].w[r & 1] * ax[1].w[r >> 1];
#pragma unroll
            for (int k = 0; k < NC; ++k)
                g[k] = fmaf(f, fmaf(m[1][k], ax[2].w[1], m[0][k] * ax[2].w[0]), g[k]);
        }
#pragma unroll
        for (int k = 0; k < NC; ++k) out[q * NC + k] = __fadd_rn(v[k], g[k]);
    }
}

template <int NC>
__global__ void __launch_bounds__(256) k_gather_adj_cic(Cic p, const int16_t *__restrict__ pmid,
                                                        const float *__restrict__ disp, int64_t n,
                                                        const float *__restrict__ mesh,
                                                        const float *__restrict__ val_cot,
                                                        float *disp_cot, float *mesh_cot) {
    for (int64_t q0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); q0 < n;
         q0 += (int64_t)gridDim.x * blockDim.x) {   // warp-uniform
        const int64_t q = q0 + (threadIdx.x & 31);
        CicAxis ax[3] = {};
        float v[NC] = {};
        if (q < n) {
            float c[3] = {0.f, 0.f, 0.f};
            cic_axes(p, pmid, disp, q, ax);
            ld_val<NC>(val_cot, 0.f, q, v);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float m[2][NC], t[2] = {0.f, 0.f};
                cic_read<NC>(p, ax, r, mesh, m);
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    t[0] = fmaf(m[0][k], v[k], t[0]);
                    t[1] = fmaf(m[1][k], v[k], t[1]);
                }
                cic_grad(ax, r, t, c);
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) disp_cot[3 * q + a] = div_or_mul(c[a], p.div, p.div_inv);
        }
        cic_add<NC>(p, q < n, ax, v, mesh_cot);
    }
}

// Whether the k_*_cic kernels cover this enmesh: 3-D, the default branch,
// periodic, every wrapped neighbour inside the mesh array, 32-bit offsets.
// mesh is the array that is added to (NULL: only read), n particles.
static bool cic_params(const EmParams &e, int64_t chan, int64_t n, const float *mesh, Cic *p) {
    if (e.dim != 3 || e.f64 || (chan != 1 && chan != 3)) return false;
    for (int a = 0; a < 3; ++a)
        if (e.wrap[a] <= 0 || e.shape[a] < e.wrap[a]) return false;
    if (e.stride[0] * chan >= (int64_t)1 << 32) return false;
    for (int a = 0; a < 3; ++a) {
        p->wrap[a] = e.wrap[a];
        p->i12[a] = e.i12[a];
        p->d12[a] = e.d12[a];
    }
    p->cell = e.cellf;
    p->inv = e.cell_inv;
    p->div = e.cot_div;
    p->div_inv = exact_inverse(e.cot_div);
    p->s0 = e.stride[0];
    p->s1 = (unsigned)e.stride[1];
    p->join = (int64_t)e.wrap[0] * e.wrap[1] * e.wrap[2] < 4 * n;
    p->pair = (uintptr_t)mesh % 8 == 0;
    return true;
}

// Blocks of a particle kernel: one particle per thread.  Short blocks are
// replaced as they end, where a few long ones hold their share of the particles
// up behind contended reductions.
static int ptcl_blocks(int64_t n, int threads) {
    const int64_t g = (n + threads - 1) / threads;
    return (int)(g < (1 << 30) ? g : 1 << 30);
}

}  // namespace pmx

using namespace pmx;

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------

extern "C" int pmx_version(void) { return 200; }

extern "C" const char *pmx_last_error(void) { return g_err.c_str(); }

extern "C" int pmx_device_sms(int *sms) {
    if (!sms) return fail(PMX_ERR_ARG, "null sms");
    *sms = device_sms();
    return PMX_OK;
}

extern "C" int pmx_stream_create(int device, void **stream) {
    if (!stream) return fail(PMX_ERR_ARG, "null stream");
    *stream = nullptr;
    int prev = 0;
    PMX_CUDA(cudaGetDevice(&prev));
    PMX_CUDA(cudaSetDevice(device));
    cudaStream_t s = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    cudaSetDevice(prev);
    if (e != cudaSuccess) return cuda_status(e, "cudaStreamCreateWithFlags");
    *stream = reinterpret_cast<void *>(s);
    return PMX_OK;
}

extern "C" int pmx_stream_destroy(void *stream) {
    if (!stream) return PMX_OK;
    PMX_CUDA(cudaStreamDestroy(reinterpret_cast<cudaStream_t>(stream)));
    return PMX_OK;
}

static int check_common(const pmx_enmesh_spec *spec, const void *pmid, const void *disp,
                        int64_t n, EmParams *p) {
    int st = make_em_params(spec, p);
    if (st) return st;
    if (n < 0) return fail(PMX_ERR_ARG, "negative particle count");
    if (n > 0 && (!pmid || !disp)) return fail(PMX_ERR_ARG, "null pmid/disp");
    return PMX_OK;
}

extern "C" int pmx_enmesh(const pmx_enmesh_spec *spec, const int16_t *pmid, const float *disp,
                          int64_t n, int32_t *ind, float *frac, float *frac_grad, void *stream) {
    EmParams p;
    int st = check_common(spec, pmid, disp, n, &p);
    if (st) return st;
    if (n == 0) return PMX_OK;
    if (!frac) return fail(PMX_ERR_ARG, "null frac");
    const int T = 256;
    k_enmesh<<<stride_grid(n, T), T, 0, as_stream(stream)>>>(p, pmid, disp, n, ind, frac, frac_grad);
    PMX_LAUNCH_CHECK("k_enmesh");
    return PMX_OK;
}

extern "C" int pmx_scatter(const pmx_enmesh_spec *spec, const int16_t *pmid, const float *disp,
                           int64_t n, const float *val, float val_scalar, int64_t channels,
                           float *mesh, void *stream) {
    EmParams p;
    int st = check_common(spec, pmid, disp, n, &p);
    if (st) return st;
    if (channels < 1) return fail(PMX_ERR_ARG, "channels must be >= 1");
    if (!val && channels != 1) return fail(PMX_ERR_SHAPE, "scalar val needs channels == 1");
    if (!mesh) return fail(PMX_ERR_ARG, "null mesh");
    if (n == 0) return PMX_OK;
    const int T = 256;
    Cic q;
    if (cic_params(p, channels, n, mesh, &q))
        (channels == 1 ? k_scatter_cic<1> : k_scatter_cic<3>)
            <<<ptcl_blocks(n, T), T, 0, as_stream(stream)>>>(q, pmid, disp, n, val, val_scalar, mesh);
    else
        k_scatter<<<ptcl_blocks(n, T), T, 0, as_stream(stream)>>>(p, pmid, disp, n, val, val_scalar,
                                                                  channels, mesh);
    PMX_LAUNCH_CHECK("k_scatter");
    return PMX_OK;
}

extern "C" int pmx_scatter_adj(const pmx_enmesh_spec *spec, const int16_t *pmid,
                               const float *disp, int64_t n, const float *val, float val_scalar,
                               int64_t channels, const float *mesh_cot, float *disp_cot,
                               float *val_cot, void *stream) {
    EmParams p;
    int st = check_common(spec, pmid, disp, n, &p);
    if (st) return st;
    if (channels < 1) return fail(PMX_ERR_ARG, "channels must be >= 1");
    if (!val && channels != 1) return fail(PMX_ERR_SHAPE, "scalar val needs channels == 1");
    if (!mesh_cot || (n > 0 && !disp_cot)) return fail(PMX_ERR_ARG, "null mesh_cot/disp_cot");
    if (n == 0) return PMX_OK;
    const int T = 256;
    Cic q;
    if (cic_params(p, channels, n, nullptr, &q))
        (channels == 1 ? k_scatter_adj_cic<1> : k_scatter_adj_cic<3>)
            <<<ptcl_blocks(n, T), T, 0, as_stream(stream)>>>(q, pmid, disp, n, val, val_scalar,
                                                             mesh_cot, disp_cot, val_cot);
    else
        k_scatter_adj<<<ptcl_blocks(n, T), T, 0, as_stream(stream)>>>(
            p, pmid, disp, n, val, val_scalar, channels, mesh_cot, disp_cot, val_cot);
    PMX_LAUNCH_CHECK("k_scatter_adj");
    return PMX_OK;
}

extern "C" int pmx_gather(const pmx_enmesh_spec *spec, const int16_t *pmid, const float *disp,
                          int64_t n, const float *mesh, int64_t channels, const float *val,
                          float val_scalar, float *out, void *stream) {
    EmParams p;
    int st = check_common(spec, pmid, disp, n, &p);
    if (st) return st;
    if (channels < 1) return fail(PMX_ERR_ARG, "channels must be >= 1");
    if (!mesh || (n > 0 && !out)) return fail(PMX_ERR_ARG, "null mesh/out");
    if (n == 0) return PMX_OK;
    const int T = 256;
    Cic q;
    if (cic_params(p, channels, n, nullptr, &q))
        (channels == 1 ? k_gather_cic<1> : k_gather_cic<3>)
            <<<ptcl_blocks(n, T), T, 0, as_stream(stream)>>>(q, pmid, disp, n, mesh, val, val_scalar,
                                                             out);
    else
        k_gather<<<ptcl_blocks(n, T), T, 0, as_stream(stream)>>>(p, pmid, disp, n, mesh, channels,
                                                                 val, val_scalar, out);
    PMX_LAUNCH_CHECK("k_gather");
    return PMX_OK;
}

extern "C" int pmx_gather_adj(const pmx_enmesh_spec *spec, const int16_t *pmid,
                              const float *disp, int64_t n, const float *mesh, int64_t channels,
                              const float *val_cot, float *disp_cot, float *mesh_cot,
                              void *stream) {
    EmParams p;
    int st = check_common(spec, pmid, disp, n, &p);
    if (st) return st;
    if (channels < 1) return fail(PMX_ERR_ARG, "channels must be >= 1");
    if (!mesh || !mesh_cot || (n > 0 && (!val_cot || !disp_cot)))
        return fail(PMX_ERR_ARG, "null mesh/mesh_cot/val_cot/disp_cot");
    if (n == 0) return PMX_OK;
    const int T = 256;
    Cic q;
    if (cic_params(p, channels, n, mesh_cot, &q))
        (channels == 1 ? k_gather_adj_cic<1> : k_gather_adj_cic<3>)
            <<<ptcl_blocks(n, T), T, 0, as_stream(stream)>>>(q, pmid, disp, n, mesh, val_cot,
                                                             disp_cot, mesh_cot);
    else
        k_gather_adj<<<ptcl_blocks(n, T), T, 0, as_stream(stream)>>>(
            p, pmid, disp, n, mesh, channels, val_cot, disp_cot, mesh_cot);
    PMX_LAUNCH_CHECK("k_gather_adj");
    return PMX_OK;
}
