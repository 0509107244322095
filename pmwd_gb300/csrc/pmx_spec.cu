// Power-spectrum binning of half spectra (pmwd/spec_util.py:50-147).
//
// The reference builds |k|, P and the Hermitian multiplicity as full-mesh
// float64 arrays, digitizes |k| against the bin edges and sums with
// bincount.  Here one pass reads the complex64 spectrum (and the second one
// of a cross spectrum) once: every thread computes |k| from the float64
// wavenumber tables in the reference's order ((kx^2 + ky^2) + kz^2), the bin
// with numpy digitize semantics, P in float64 (|F|^2 from the widened parts,
// or F conj(G) formed in complex64 and widened, as the reference does), the
// optional sinc^-deconv window, and accumulates k N, P N and N per bin: sums of
// each thread's run of cells, then shared-memory float64 sums merged once per
// block.

#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <climits>

#include "pmx_internal.cuh"

namespace pmx {
namespace {

constexpr int ST = 256;
constexpr int SMEM_BINS = 2048;  // per-block shared accumulators up to this many bins

// numpy.digitize(x, edges, right): right = 0 -> count of edges <= x,
// right = 1 -> count of edges < x (edges increasing).
__device__ __forceinline__ int digitize(double x, const double *e, int ne, int right) {
    int lo = 0, hi = ne;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const bool go = right ? (e[mid] < x) : (e[mid] <= x);
        if (go) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// sinc(x) = sin(pi x) / (pi x), 1 at 0 (torch.sinc / jnp.sinc)
__device__ __forceinline__ double sincd(double x) {
    return x == 0.0 ? 1.0 : sinpi(x) / (3.141592653589793238462643383279502884 * x);
}

struct SpecArgs {
    const float2 *F, *G;
    int64_t nb, n0, n1, n2h, Mc;
    int nyq_z;                    // 1: the last z index is the Nyquist plane (even n2)
    const double *kx, *ky, *kz;   // cycles per sample (fftfreq / rfftfreq)
    const long long *keys;        // k_edge_keys
    int ne, nbin;
    const double *wx, *wy, *wz;   // sinc^-deconv per axis, or NULL
    double *ksum, *psum, *nsum;   // nbin, 2 nbin (re, im), nbin
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The order of nonnegative doubles is that of their bits.  keys[b] is the
// smallest s with sqrt(s) beyond edge b (sqrt(s) >= e, or > e with right): |k| is
// beyond the edge exactly where |k|^2 >= keys[b], rounding of the root included.
__global__ void k_edge_keys(const double *edges, int ne, int right, long long *keys) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= ne) return;
    const double e = edges[b];
    auto beyond = [&](long long s) {
        const double k = sqrt(__longlong_as_double(s));
        return right ? k > e : k >= e;
    };
    const long long inf = 0x7ff0000000000000ll;
    long long s = LLONG_MAX;   // e NaN, or its square above every float64
    if (e < 0.0 || (e == 0.0 && !right)) {
        s = 0;
    } else if (e * e < __longlong_as_double(inf)) {
        s = __double_as_longlong(e * e);
        // the square and the root round: a few steps either way
        for (int i = 0; i < 8 && s > 0 && beyond(s - 1); ++i) --s;
        for (int i = 0; i < 8 && s < inf && !beyond(s); ++i) ++s;
    }
    keys[b] = s;
}

// Root of s >= 0 by Heron steps k + (s - k^2) / (2 k) from the float32 unit's
// reciprocal root: two steps leave the rounding of the last one.
__device__ __forceinline__ double root(double s) {
    const unsigned hi = (unsigned)__double2hiint(s);
    if (hi < 0x3c900000u || hi >= 0x43000000u) return sqrt(s);   // outside 2^-54 .. 2^49
    // s truncated to float32, by the exponent and the upper mantissa bits
    const float f = __uint_as_float(((hi - 0x38000000u) << 3) |
                                    ((unsigned)__double2loint(s) >> 29));
    const float r = rsqrtf(f);
    const double h = to_f64(0.5f * r);
    double k = to_f64(f * r);
    k = fma(fma(-k, k, s), h, k);
    return fma(fma(-k, k, s), h, k);
}

// A warp takes consecutive rows, (x, y) along kz or with ZM (kz, x) along y, and
// each lane a contiguous run of their cells: the lane keeps the sums of its
// current bin in registers, steps through the edges as |k| passes them, and adds
// its sums to the block's shared accumulators (SH) or to global memory when the
// bin changes.  The float64 unit is the bound (one to two operations per clock
// and SM), so x and y run over half their indices only: the up to four cells at
// +-kx, +-ky have one |k|, root, bin and window.  Bins come from integer
// comparisons, the windows (three powers of sines per cell before) from tables
// per axis, and the multiplicity 2 from one doubling per flush.  462^3, log bins:
// 0.99 ms (5.2 with a binary search, a root and two widened products per cell);
// 347^3, bins of the fundamental width, window: 0.53 (27).
template <bool SH, bool ZM>
__global__ void __launch_bounds__(ST) k_powspec(SpecArgs a) {
    extern __shared__ double sb[];  // SH: 4 doubles per bin (k N, P_re N, P_im N, N)
    if (SH) {
        for (int i = threadIdx.x; i < 4 * a.nbin; i += ST) sb[i] = 0.0;
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const int n0 = (int)a.n0, n1 = (int)a.n1, n2h = (int)a.n2h;
    const int m0 = n0 / 2 + 1, m1 = n1 / 2 + 1, len = ZM ? m1 : n2h;
    const int64_t rows = (int64_t)m0 * (ZM ? n2h : m1), nw = (int64_t)gridDim.x * (ST / 32);
    const int run = (len + 31) / 32, c0 = lane * run, c1 = c0 + run < len ? c0 + run : len;
    const int64_t per = (rows + nw - 1) / nw;
    const int64_t r0 = ((int64_t)blockIdx.x * (ST / 32) + (threadIdx.x >> 5)) * per;
    const int64_t r1 = r0 + per < rows ? r0 + per : rows;
    double sk = 0.0, sp = 0.0, si = 0.0;   // half the sums of k N, P N
    int cnt = 0, b = -1;
    long long lo = 0, hi = -1;             // keys of bin b's lower edge and of the next
    auto flush = [&]() {
        if (cnt == 0) return;
        double *k = SH ? sb + 4 * b : a.ksum + b, *p = SH ? sb + 4 * b + 1 : a.psum + 2 * b;
        atomicAdd(k, sk + sk);
        atomicAdd(p, sp + sp);
        if (a.G) atomicAdd(p + 1, si + si);
        atomicAdd(SH ? sb + 4 * b + 3 : a.nsum + b, (double)cnt);
        sk = sp = si = 0.0;
        cnt = 0;
    };
    for (int64_t row = r0; row < r1; ++row) {
        const int jl = (int)(row / m0), i = (int)(row - (int64_t)jl * m0);   // ky or kz; x
        const int i2 = n0 - i;
        const bool xx = i > 0 && i2 > i;   // -kx is another cell
        const double kx = a.kx[i], kr = ZM ? a.kz[jl] : a.ky[jl];
        const double kx2 = __dmul_rn(kx, kx), kr2 = __dmul_rn(kr, kr);
        const double kxy = ZM ? kx2 : __dadd_rn(kx2, kr2);
        const double wr = a.wx ? ZM ? a.wx[i] : a.wx[i] * a.wy[jl] : 1.0;
        for (int c = c0; c < c1; ++c) {
            const int j = ZM ? c : jl, l = ZM ? jl : c, j2 = n1 - j;
            const bool yy = j > 0 && j2 > j;
            const double kc = (ZM ? a.ky : a.kz)[c];
            double s = __dadd_rn(kxy, __dmul_rn(kc, kc));   // (kx^2 + ky^2) + kz^2
            if (ZM) s = __dadd_rn(s, kr2);
            const long long key = __double_as_longlong(s);
            if (key >= hi || key < lo) {
                flush();
                if (b < 0) {
                    int e = 0, h = a.ne;   // numpy.digitize
                    while (e < h) {
                        const int mid = (e + h) >> 1;
                        if (a.keys[mid] <= key) e = mid + 1;
                        else h = mid;
                    }
                    b = e;
                }
                while (b < a.ne && key >= a.keys[b]) ++b;
                while (b > 0 && key < a.keys[b - 1]) --b;
                lo = b > 0 ? a.keys[b - 1] : LLONG_MIN;
                hi = b < a.ne ? a.keys[b] : LLONG_MAX;
            }
            if (b >= a.nbin) continue;
            double pr = 0.0, pi = 0.0;
            auto add = [&](int x, int y) {
                const int64_t at = ZM ? ((int64_t)l * n0 + x) * n1 + y
                                      : ((int64_t)x * n1 + y) * n2h + l;
                for (int64_t t = 0; t < a.nb; ++t) {
                    const float2 f = a.F[t * a.Mc + at];
                    if (a.G) {
                        const float2 gg = a.G[t * a.Mc + at];
                        // F * conj(G) in complex64, then widened
                        pr += to_f64(__fadd_rn(__fmul_rn(f.x, gg.x), __fmul_rn(f.y, gg.y)));
                        pi += to_f64(__fsub_rn(__fmul_rn(f.y, gg.x), __fmul_rn(f.x, gg.y)));
                    } else {
                        const double x = to_f64(f.x), y = to_f64(f.y);
                        pr = fma(y, y, fma(x, x, pr));
                    }
                }
            };
            add(i, j);
            if (xx) add(i2, j);
            if (yy) add(i, j2);
            if (xx && yy) add(i2, j2);
            if (a.wx) {
                const double w = ZM ? (wr * a.wy[c]) * a.wz[jl] : wr * a.wz[c];
                pr *= w;
                pi *= w;
            }
            const double k = root(s);
            const int cells = (xx ? 2 : 1) * (yy ? 2 : 1);
            const bool one = l == 0 || (a.nyq_z && l == n2h - 1);
            if (one) {
                pr *= 0.5;
                pi *= 0.5;
            }
            const int N = one ? cells : 2 * cells;
            sk = fma(k, 0.5 * N, sk);
            sp += pr;
            if (a.G) si += pi;
            cnt += N;
        }
    }
    flush();
    if (SH) {
        __syncthreads();
        for (int b = threadIdx.x; b < a.nbin; b += ST) {
            if (sb[4 * b + 3] == 0.0) continue;
            atomicAdd(a.ksum + b, sb[4 * b]);
            atomicAdd(a.psum + 2 * b, sb[4 * b + 1]);
            if (a.G) atomicAdd(a.psum + 2 * b + 1, sb[4 * b + 2]);
            atomicAdd(a.nsum + b, sb[4 * b + 3]);
        }
    }
}

// ---------------------------------------------------------------------------
// Power-of-two grids.  fftfreq values are i/n exactly, so k^2 = i^2/n0^2 +
// j^2/n1^2 + l^2/n2^2 is exact in float64 (multiples of 1/D, D = max(n)^2)
// whatever the summation order, and k = sqrt(m / D) with the integer
// m = i^2 D/n0^2 + j^2 D/n1^2 + l^2 D/n2^2: |k| and its bin depend on m only.
// Tables of k(m) and bin(m) (built once per call, float64 as the reference)
// replace the per-cell float64 |k|.  GB300's float64 rate is low, so this
// path keeps float64 out of the per-cell work: P N is formed in float32 and
// summed per bin with warp shuffles before one float64 add.  The sums k N
// and N depend on the grid alone; they are accumulated (float64 per cell)
// only when ksum / nsum are given, so a caller can compute them once per
// grid and bins and pass NULL afterwards.
// ---------------------------------------------------------------------------

struct Pow2Args {
    const float2 *F, *G;
    int64_t nb, n0, n1, n2h, Mc;
    int nyq_z;
    int64_t ax, ay, az;            // D / n_a^2
    int h0, h1;                    // n0, n1 (signed index: i' = i <= n/2 ? i : i - n)
    const double *ktab;            // k(m)
    const int *btab;               // bin(m), nbin = none
    const int *thr;                // k_thresholds, instead of bin(m)
    const float *wx, *wy, *wz;     // sinc^-deconv per axis, or NULL
    int nbin;
    int zm;                        // 1: layout (n2h, n0, n1), y contiguous
    double *ksum, *psum, *nsum;
};

__global__ void k_pow2_tables(int64_t mmax, double D, const double *edges, int ne, int right,
                              int nbin, double *ktab, int *btab) {
    for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m <= mmax;
         m += (int64_t)gridDim.x * blockDim.x) {
        const double k = sqrt((double)m / D);  // exact quotient (D a power of two)
        ktab[m] = k;
        if (!btab) continue;
        const int b = digitize(k, edges, ne, right);
        btab[m] = b < nbin ? b : nbin;
    }
}

__device__ __forceinline__ float warp_sumf(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One warp per (x, y) row of n2h cells, lanes on consecutive kz (coalesced
// loads); per 32 cells, shuffle sums per distinct bin (usually one or two)
// and one float64 shared-memory add per bin.  CROSS: F conj(G); GEOM: also
// the sums of k N and N; WIN: sinc^-deconv windows.  PRIV (few bins): every
// warp owns its own bin array, so the per-bin adds are plain stores of one
// lane instead of float64 atomics that all warps of the block contend for;
// the arrays are summed at the end.
constexpr int PRIV_BINS = 64;

template <bool CROSS, bool GEOM, bool WIN, bool PRIV>
__global__ void __launch_bounds__(ST, 6) k_powspec_rows(Pow2Args a) {
    extern __shared__ double sbase[];  // 4 doubles per bin (per warp with PRIV)
    const int nacc = (PRIV ? ST / 32 : 1) * 4 * a.nbin;
    for (int i = threadIdx.x; i < nacc; i += ST) sbase[i] = 0.0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    double *sb = PRIV ? sbase + (threadIdx.x >> 5) * 4 * a.nbin : sbase;
    const int n2h = (int)a.n2h, az = (int)a.az;
    // rows of contiguous cells: (x, y) rows along kz for the (n0, n1, n2h)
    // layout; with zm, (kz, x) rows along y of the (n2h, n0, n1) layout that
    // torch's CUDA rfftn returns, which this kernel serves only for n1 < 32
    // or n1 not a multiple of 32 (k_powspec_runs takes the others)
    // every index below fits in 32 bits (grids up to 2048: rows < 2^22,
    // bin-table indices < 2^31)
    const int n0 = (int)a.n0, n1 = (int)a.n1, h0 = a.h0, h1 = a.h1;
    const int ax = (int)a.ax, ay = (int)a.ay;
    const int nrows = a.zm ? n2h * n0 : n0 * n1;
    const int nlane = a.zm ? n1 : n2h;
    const int wstride = gridDim.x * (ST / 32);
    for (int row = blockIdx.x * (ST / 32) + (threadIdx.x >> 5); row < nrows;
         row += wstride) {  // warp-uniform
        int i, j = 0, lr = 0, mrow;
        if (a.zm) {
            lr = row / n0;
            i = row - lr * n0;
            const int si = i <= h0 / 2 ? i : i - h0;
            mrow = si * si * ax + lr * lr * az;
        } else {
            i = row / n1;
            j = row - i * n1;
            const int si = i <= h0 / 2 ? i : i - h0, sj = j <= h1 / 2 ? j : j - h1;
            mrow = si * si * ax + sj * sj * ay;
        }
        const float2 *Fr = a.F + (int64_t)row * nlane;
        const float2 *Gr = CROSS ? a.G + (int64_t)row * nlane : nullptr;
        for (int c0 = 0; c0 < nlane; c0 += 32) {
            const int c = c0 + lane;   // kz, or y with zm
            int b = a.nbin;
            float pr = 0.f, pi = 0.f;
            double kn = 0.0, nn = 0.0;
            if (c < nlane) {
                int m, l, jj;
                if (a.zm) {
                    const int sjj = c <= h1 / 2 ? c : c - h1;
                    m = mrow + sjj * sjj * ay;
                    l = lr;
                    jj = c;
                } else {
                    m = mrow + c * c * az;
                    l = c;
                    jj = j;
                }
                b = a.btab[m];
                if (b < a.nbin) {
                    for (int64_t t = 0; t < a.nb; ++t) {
                        const float2 f = Fr[t * a.Mc + c];
                        if (CROSS) {
                            const float2 gg = Gr[t * a.Mc + c];
                            pr += __fadd_rn(__fmul_rn(f.x, gg.x), __fmul_rn(f.y, gg.y));
                            pi += __fsub_rn(__fmul_rn(f.y, gg.x), __fmul_rn(f.x, gg.y));
                        } else {
                            pr += fmaf(f.x, f.x, f.y * f.y);
                        }
                    }
                    if (WIN) {  // ((P wx) wy) wz
                        const float w = (a.wx[i] * a.wy[jj]) * a.wz[l];
                        pr *= w;
                        pi *= w;
                    }
                    const bool two = !(l == 0 || (a.nyq_z && l == n2h - 1));
                    if (two) {
                        pr += pr;
                        pi += pi;
                    }
                    if (GEOM) {
                        const double k = a.ktab[m];
                        kn = two ? k + k : k;
                        nn = two ? 2.0 : 1.0;
                    }
                }
            }
            // many distinct bins in these 32 cells (fine linear bins): each
            // lane adds its own values; few: shuffle sums per bin
            const unsigned peers = __match_any_sync(0xffffffffu, b);
            const int ndist = __popc(__ballot_sync(0xffffffffu, lane == __ffs(peers) - 1));
            if (ndist > 4) {
                if (b < a.nbin) {
                    atomicAdd(sb + 4 * b + 1, (double)pr);
                    if (CROSS) atomicAdd(sb + 4 * b + 2, (double)pi);
                    if (GEOM) {
                        atomicAdd(sb + 4 * b, kn);
                        atomicAdd(sb + 4 * b + 3, nn);
                    }
                }
                continue;
            }
            unsigned pending = __ballot_sync(0xffffffffu, b < a.nbin);
            while (pending) {
                const int src = __ffs(pending) - 1;
                const int bb = __shfl_sync(0xffffffffu, b, src);
                const bool mine = b == bb;
                const float spr = warp_sumf(mine ? pr : 0.f);
                const float spi = CROSS ? warp_sumf(mine ? pi : 0.f) : 0.f;
                double sk = 0.0, sn = 0.0;
                if (GEOM) {
                    sk = warp_sum(mine ? kn : 0.0);
                    sn = warp_sum(mine ? nn : 0.0);
                }
                if (lane == src) {
                    if (PRIV) {  // this warp's array: one lane at a time
                        sb[4 * bb + 1] += (double)spr;
                        if (CROSS) sb[4 * bb + 2] += (double)spi;
                        if (GEOM) {
                            sb[4 * bb] += sk;
                            sb[4 * bb + 3] += sn;
                        }
                    } else {
                        atomicAdd(sb + 4 * bb + 1, (double)spr);
                        if (CROSS) atomicAdd(sb + 4 * bb + 2, (double)spi);
                        if (GEOM) {
                            atomicAdd(sb + 4 * bb, sk);
                            atomicAdd(sb + 4 * bb + 3, sn);
                        }
                    }
                }
                pending &= ~__ballot_sync(0xffffffffu, mine);
            }
            if (PRIV) __syncwarp();  // the next chunk's adds see these
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < a.nbin; b += ST) {
        double acc[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] = sbase[4 * b + c];
        if (PRIV)
            for (int w = 1; w < ST / 32; ++w)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[c] += sbase[w * 4 * a.nbin + 4 * b + c];
        if (GEOM) {
            atomicAdd(a.ksum + b, acc[0]);
            atomicAdd(a.nsum + b, acc[3]);
        }
        atomicAdd(a.psum + 2 * b, acc[1]);
        if (CROSS) atomicAdd(a.psum + 2 * b + 1, acc[2]);
    }
}

// Half-axis-major spectra with n1 a multiple of 32.  A warp takes units of up to
// 512 consecutive y cells of a row (kz, x), stages them in shared memory with
// coalesced loads, and lane r walks the run of R = cells / 32 cells from r R,
// keeping the sums of its current bin in registers until the bin changes, across
// units too.  The bins are shells in |k|, hence intervals [T[b], T[b+1]) of the
// integer m: comparing m with the current interval's ends replaces a table
// lookup per cell.  512^3, log bins, window: 0.32 ms (0.59 with each lane reading
// its run from global memory, a bin lookup and a float64 addition per cell);
// reading the spectrum alone takes 0.08, the rest is instructions and the wait
// for the next unit's loads.
constexpr int UNIT = 512;

template <bool CROSS, bool GEOM, bool WIN, bool PRIV, bool ONE>
__global__ void __launch_bounds__(ST, 6) k_powspec_runs(Pow2Args a) {
    extern __shared__ double sbase[];  // 4 doubles per bin (per warp with PRIV), then T and the rows
    const int nbin = a.nbin, nacc = (PRIV ? ST / 32 : 1) * 4 * nbin;
    int *T = reinterpret_cast<int *>(sbase + nacc);
    const int n2h = (int)a.n2h, n0 = (int)a.n0, n1 = (int)a.n1, h0 = a.h0, h1 = a.h1;
    const int cells = n1 < UNIT ? n1 : UNIT, R = cells / 32, U = n1 / cells;
    const int rsh = __ffs(R) - 1, rowlen = cells + 32;   // one pad per run
    float *rows = reinterpret_cast<float *>(T + ((nbin + 2 + 3) & ~3));
    for (int i = threadIdx.x; i < nacc; i += ST) sbase[i] = 0.0;
    for (int i = threadIdx.x; i < nbin + 2; i += ST) T[i] = a.thr[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *sb = PRIV ? sbase + warp * 4 * nbin : sbase;
    float *Ps = rows + warp * (CROSS ? 2 : 1) * rowlen, *Qs = Ps + rowlen;   // P N: re, im
    const int ax = (int)a.ax, ay = (int)a.ay, az = (int)a.az;
    // consecutive units per warp, so that a lane's bin hardly moves between them
    // (of rows longer than a unit, first all their first units, and so on)
    const int nrows = n2h * n0;
    const int64_t units = (int64_t)nrows * U, nw = (int64_t)gridDim.x * (ST / 32);
    const int64_t per = (units + nw - 1) / nw, w = (int64_t)blockIdx.x * (ST / 32) + warp;
    const int64_t u0 = w * per, u1 = u0 + per < units ? u0 + per : units;
    int cur = 0, lo = T[0];
    unsigned width = (unsigned)(T[1] - lo);
    double ar = 0.0, ai = 0.0, ak = 0.0;
    int an = 0;
    // A bin's cells within a run: float32 sums with the rounding errors of their
    // additions summed beside, some 2^-46 of the sum, in place of a float64
    // addition per cell (about 30 clocks of the float64 unit per warp).
    float gr = 0.f, er = 0.f, gi = 0.f, ei = 0.f;
    auto add2 = [](float &s, float &e, float p) {
        const float t = __fadd_rn(s, p), q = __fsub_rn(t, s);
        e = __fadd_rn(e, __fadd_rn(__fsub_rn(s, __fsub_rn(t, q)), __fsub_rn(p, q)));
        s = t;
    };
    auto fold = [&](const float *P, const float *Q, int n) {   // the last n cells before P, Q
        if (n == 0) return;
        // beyond float32: cell by cell
        if (fabsf(gr) <= FLT_MAX && fabsf(gi) <= FLT_MAX) {
            ar += to_f64(gr) + to_f64(er);
            if (CROSS) ai += to_f64(gi) + to_f64(ei);
        } else {
            for (int c = -n; c < 0; ++c) {
                ar += (double)P[c];
                if (CROSS) ai += (double)Q[c];
            }
        }
        gr = er = gi = ei = 0.f;
    };
    auto flush = [&]() {
        if (cur < nbin) {
            atomicAdd(sb + 4 * cur + 1, ar);
            if (CROSS) atomicAdd(sb + 4 * cur + 2, ai);
            if (GEOM) {
                atomicAdd(sb + 4 * cur, ak);
                atomicAdd(sb + 4 * cur + 3, (double)an);
            }
        }
        ar = ai = ak = 0.0;
        an = 0;
    };
    for (int64_t u = u0; u < u1; ++u) {
        const int sub = (int)(u / nrows), row = (int)(u - (int64_t)sub * nrows);
        const int l = row / n0, i = row - l * n0, si = i <= h0 / 2 ? i : i - h0;
        const int mrow = si * si * ax + l * l * az;
        const bool two = !(l == 0 || (a.nyq_z && l == n2h - 1));
        const float wxi = WIN ? a.wx[i] : 1.f, wzl = WIN ? a.wz[l] : 1.f;
        const int64_t base = (int64_t)row * n1 + sub * cells;
        __syncwarp();   // the previous unit's reads
#pragma unroll 4
        for (int c = lane; c < cells; c += 32) {
            float pr = 0.f, pi = 0.f;
            const float2 *Fc = a.F + base + c, *Gc = CROSS ? a.G + base + c : nullptr;
            int64_t t = a.nb;
            do {
                const float2 f = *Fc;
                if (CROSS) {
                    const float2 gg = *Gc;
                    pr += __fadd_rn(__fmul_rn(f.x, gg.x), __fmul_rn(f.y, gg.y));
                    pi += __fsub_rn(__fmul_rn(f.y, gg.x), __fmul_rn(f.x, gg.y));
                    Gc += a.Mc;
                } else {
                    pr += fmaf(f.x, f.x, f.y * f.y);
                }
                Fc += a.Mc;
            } while (!ONE && --t > 0);
            if (WIN) {  // ((P wx) wy) wz
                const float wt = (wxi * a.wy[sub * cells + c]) * wzl;
                pr *= wt;
                pi *= wt;
            }
            if (two) {
                pr += pr;
                pi += pi;
            }
            Ps[c + (c >> rsh)] = pr;
            if (CROSS) Qs[c + (c >> rsh)] = pi;
        }
        __syncwarp();
        // R divides n1 / 2 (or is 1): |ky| rises or falls along the whole run
        const float *P = Ps + lane * (R + 1), *Q = Qs + lane * (R + 1);
        const int j0 = sub * cells + lane * R, up = j0 < h1 / 2 ? 1 : -1, y0 = up > 0 ? j0 : h1 - j0;
        int m = mrow + y0 * y0 * ay, dm = (2 * up * y0 + 1) * ay, from = 0;
#pragma unroll 4
        for (int r = 0; r < R; ++r) {
            if ((unsigned)(m - lo) >= width) {
                fold(P + r, Q + r, r - from);
                from = r;
                flush();
                while (m >= T[cur + 1]) ++cur;   // T[nbin + 1] is above every m
                while (m < T[cur]) --cur;        // and T[0] below
                lo = T[cur];
                width = (unsigned)(T[cur + 1] - lo);
            }
            add2(gr, er, P[r]);
            if (CROSS) add2(gi, ei, Q[r]);
            if (GEOM) {
                const double k = a.ktab[m];
                ak += two ? k + k : k;
                an += two ? 2 : 1;
            }
            m += dm;
            dm += 2 * ay;
        }
        fold(P + R, Q + R, R - from);
    }
    flush();
    __syncthreads();
    for (int b = threadIdx.x; b < nbin; b += ST) {
        double acc[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] = sbase[4 * b + c];
        if (PRIV)
            for (int w2 = 1; w2 < ST / 32; ++w2)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[c] += sbase[w2 * 4 * nbin + 4 * b + c];
        if (GEOM) {
            atomicAdd(a.ksum + b, acc[0]);
            atomicAdd(a.nsum + b, acc[3]);
        }
        atomicAdd(a.psum + 2 * b, acc[1]);
        if (CROSS) atomicAdd(a.psum + 2 * b + 1, acc[2]);
    }
}

// Dynamic shared memory above the default 48 KB needs the opt-in attribute.
template <class K>
void allow_smem(K *kern, size_t sm) {
    if (sm > 48 * 1024)
        cudaFuncSetAttribute(reinterpret_cast<const void *>(kern),
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
}

// Blocks of ST threads that an SM holds.
template <class K>
int resident(K *kern, size_t sm) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, ST, sm) != cudaSuccess || n < 1)
        n = 1;
    return n;
}

template <bool CROSS, bool GEOM, bool PRIV>
void launch_rows_p(const Pow2Args &p, cudaStream_t s) {
    size_t sm = (PRIV ? ST / 32 : 1) * 4 * (size_t)p.nbin * sizeof(double);
    if (p.thr) {   // contiguous runs per lane
        const int64_t cells = p.n1 < UNIT ? p.n1 : UNIT;
        sm += ((p.nbin + 2 + 3) & ~3) * sizeof(int) +
              ST / 32 * (CROSS ? 2 : 1) * (cells + 32) * sizeof(float);
        auto *kern = p.nb == 1 ? p.wx ? k_powspec_runs<CROSS, GEOM, true, PRIV, true>
                                      : k_powspec_runs<CROSS, GEOM, false, PRIV, true>
                               : p.wx ? k_powspec_runs<CROSS, GEOM, true, PRIV, false>
                                      : k_powspec_runs<CROSS, GEOM, false, PRIV, false>;
        allow_smem(kern, sm);
        // every warp has the same share: one wave of resident blocks
        const int grid = stride_grid(p.n2h * p.n0 * (p.n1 / cells) * 32, ST, resident(kern, sm));
        kern<<<grid, ST, sm, s>>>(p);
        return;
    }
    const int grid = stride_grid(p.n0 * p.n1 * 32, ST, 8);
    if (p.wx) {
        allow_smem(k_powspec_rows<CROSS, GEOM, true, PRIV>, sm);
        k_powspec_rows<CROSS, GEOM, true, PRIV><<<grid, ST, sm, s>>>(p);
    } else {
        allow_smem(k_powspec_rows<CROSS, GEOM, false, PRIV>, sm);
        k_powspec_rows<CROSS, GEOM, false, PRIV><<<grid, ST, sm, s>>>(p);
    }
}

template <bool CROSS, bool GEOM>
void launch_rows(const Pow2Args &p, cudaStream_t s) {
    if (p.nbin <= PRIV_BINS)
        launch_rows_p<CROSS, GEOM, true>(p, s);
    else
        launch_rows_p<CROSS, GEOM, false>(p, s);
}

// Power-of-two grids up to 2048, for which |k|^2 has an integer form.
bool pow2_grid(const int64_t n[3]) {
    for (int a = 0; a < 3; ++a)
        if (n[a] < 1 || n[a] > 2048 || (n[a] & (n[a] - 1))) return false;
    return true;
}

// sinc^-deconv of all three axes, one after the other.
struct SincArgs {
    const double *k[3];
    int n[3];
    double deconv;
};
template <typename T>
__global__ void k_sinc_tab(SincArgs s, T *w) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= s.n[0] + s.n[1] + s.n[2]) return;
    const int o = q;
    int a = 0;
    for (; a < 2 && q >= s.n[a]; ++a) q -= s.n[a];
    w[o] = (T)pow(sincd(s.k[a][q]), -s.deconv);
}

// T[b], b = 1..nbin: the smallest m <= mmax whose |k| falls into bin b or a
// later one (INT_MAX - 1: none); T[0] and T[nbin + 1] close the list.
__global__ void k_thresholds(int64_t mmax, double D, const double *edges, int right, int nbin,
                             int *T) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > nbin + 1) return;
    int t = b == 0 ? -1 : INT_MAX - 1;
    if (b >= 1 && b <= nbin) {
        const double e = edges[b - 1], g = floor(e * e * D) - 2.0;
        if (e <= 0.0 || g <= (double)mmax) {
            int64_t m = e <= 0.0 || g < 0.0 ? 0 : (int64_t)g;
            for (; m <= mmax; ++m) {
                const double k = sqrt((double)m / D);   // as k_pow2_tables
                if (right ? e < k : e <= k) {
                    t = (int)m;
                    break;
                }
            }
        }
    }
    T[b] = t;
}

// Scratch of one call: k(m), bin(m) or the thresholds and float32 windows of the
// power-of-two kernels, edge keys and float64 windows of the general one.
struct Scratch {
    bool pow2, runs;
    size_t k, b, w;   // bytes of each part, in this order
    int64_t mmax;
    size_t bytes() const { return k + b + w; }
};
Scratch scratch_of(const int64_t n[3], int32_t nedges, int32_t nbin, bool deconv, bool geom,
                   bool zm) {
    Scratch c{};
    const int64_t n2h = n[2] / 2 + 1, nwin = deconv ? n[0] + n[1] + n2h : 0;
    c.pow2 = pow2_grid(n) && nbin <= SMEM_BINS;
    if (!c.pow2) {
        c.k = (size_t)nedges * sizeof(long long);
        c.w = (size_t)nwin * sizeof(double);
        return c;
    }
    const int64_t nmax = std::max(n[0], std::max(n[1], n[2]));
    for (int a = 0; a < 3; ++a) {
        const int64_t m = n[a] / 2 * (nmax / n[a]);   // the highest frequency in units of 1 / nmax
        c.mmax += m * m;
    }
    c.runs = zm && n[1] >= 32;
    // the run kernel takes thresholds for bin(m), and k(m) only where it sums k N
    c.k = !c.runs || geom ? (size_t)(c.mmax + 1) * sizeof(double) : 0;
    c.b = (c.runs ? (size_t)nbin + 2 : (size_t)c.mmax + 1) * sizeof(int);
    c.w = (size_t)nwin * sizeof(float);
    return c;
}

// Scratch of a call whose caller brings none: stream-ordered (after a synchronisation
// that costs some 0.1 ms), given back behind the launches, also when one fails.
struct OwnScratch {
    cudaStream_t s;
    char *p = nullptr;
    int release() {
        char *q = p;
        p = nullptr;
        if (q) PMX_CUDA(cudaFreeAsync(q, s));
        return PMX_OK;
    }
    ~OwnScratch() {
        if (p) cudaFreeAsync(p, s);
    }
};

}  // namespace
}  // namespace pmx

using namespace pmx;

static int powspec_bin(const float *F, const float *G, int64_t nbatch, const int64_t grid_shape[3],
                       const double *kx, const double *ky, const double *kz, const double *edges,
                       int32_t nedges, int32_t right, int32_t nbin, double deconv, double *ksum,
                       double *psum, double *nsum, void *stream, bool zm,
                       void *scratch = nullptr) {
    clear_error();
    if (!F || !grid_shape || !kx || !ky || !kz || !edges || !psum)
        return fail(PMX_ERR_ARG, "null argument");
    if (!aligned(8, F, G) || !aligned(8, static_cast<char *>(scratch)))
        return fail(PMX_ERR_ALIGN, "spectra and scratch must be on 8 bytes");
    if (!ksum != !nsum) return fail(PMX_ERR_ARG, "ksum and nsum are both given or both NULL");
    if (nbatch < 1 || nedges < 1 || nbin < 1 || nbin > nedges)
        return fail(PMX_ERR_ARG, "need nbatch >= 1 and 1 <= nbin <= nedges");
    for (int a = 0; a < 3; ++a)
        if (grid_shape[a] < 1) return fail(PMX_ERR_SHAPE, "bad grid shape");
    SpecArgs a;
    a.F = reinterpret_cast<const float2 *>(F);
    a.G = reinterpret_cast<const float2 *>(G);
    a.nb = nbatch;
    a.n0 = grid_shape[0];
    a.n1 = grid_shape[1];
    a.n2h = grid_shape[2] / 2 + 1;
    a.Mc = a.n0 * a.n1 * a.n2h;
    a.nyq_z = grid_shape[2] % 2 == 0;
    a.kx = kx;
    a.ky = ky;
    a.kz = kz;
    a.ne = nedges;
    right = right != 0;
    a.nbin = nbin;
    a.wx = a.wy = a.wz = nullptr;
    a.ksum = ksum;
    a.psum = psum;
    a.nsum = nsum;
    cudaStream_t s = as_stream(stream);
    const int64_t nwin = deconv != 0.0 ? a.n0 + a.n1 + a.n2h : 0;
    const Scratch sc = scratch_of(grid_shape, nedges, nbin, nwin != 0, ksum != nullptr, zm);
    if (!sc.pow2 && !ksum)
        return fail(PMX_ERR_ARG, "ksum/nsum may be NULL only for power-of-two grids <= 2048");
    OwnScratch own{s};
    char *scr = static_cast<char *>(scratch);
    if (!scr) {
        PMX_CUDA(cudaMallocAsync((void **)&own.p, sc.bytes(), s));
        scr = own.p;
    }
    if (sc.pow2) {
        Pow2Args p;
        p.zm = zm;
        p.F = a.F;
        p.G = a.G;
        p.nb = a.nb;
        p.n0 = a.n0;
        p.n1 = a.n1;
        p.n2h = a.n2h;
        p.Mc = a.Mc;
        p.nyq_z = a.nyq_z;
        const int64_t nmax = std::max(grid_shape[0], std::max(grid_shape[1], grid_shape[2]));
        const int64_t D = nmax * nmax, mmax = sc.mmax;
        p.ax = D / (grid_shape[0] * grid_shape[0]);
        p.ay = D / (grid_shape[1] * grid_shape[1]);
        p.az = D / (grid_shape[2] * grid_shape[2]);
        p.h0 = (int)grid_shape[0];
        p.h1 = (int)grid_shape[1];
        p.nbin = nbin;
        p.ksum = ksum;
        p.psum = psum;
        p.nsum = nsum;
        double *ktab = reinterpret_cast<double *>(scr);
        int *bt = reinterpret_cast<int *>(scr + sc.k);
        p.ktab = ktab;
        p.btab = sc.runs ? nullptr : bt;
        p.thr = sc.runs ? bt : nullptr;
        p.wx = p.wy = p.wz = nullptr;
        if (sc.runs)
            k_thresholds<<<(nbin + 2 + 31) / 32, 32, 0, s>>>(mmax, (double)D, edges, right, nbin, bt);
        if (sc.k)
            k_pow2_tables<<<stride_grid(mmax + 1, 256, 4), 256, 0, s>>>(
                mmax, (double)D, edges, nedges, right, nbin, ktab, sc.runs ? nullptr : bt);
        if (nwin) {
            float *w = reinterpret_cast<float *>(scr + sc.k + sc.b);
            k_sinc_tab<float><<<(int)((nwin + 31) / 32), 32, 0, s>>>(
                SincArgs{{kx, ky, kz}, {(int)a.n0, (int)a.n1, (int)a.n2h}, deconv}, w);
            p.wx = w;
            p.wy = w + a.n0;
            p.wz = w + a.n0 + a.n1;
        }
        if (a.G) {
            if (ksum) launch_rows<true, true>(p, s);
            else launch_rows<true, false>(p, s);
        } else {
            if (ksum) launch_rows<false, true>(p, s);
            else launch_rows<false, false>(p, s);
        }
        PMX_LAUNCH_CHECK("k_powspec_rows");
        return own.release();
    }
    long long *keys = reinterpret_cast<long long *>(scr);
    k_edge_keys<<<(nedges + 63) / 64, 64, 0, s>>>(edges, nedges, right, keys);
    a.keys = keys;
    if (nwin) {
        double *win = reinterpret_cast<double *>(keys + nedges);
        k_sinc_tab<double><<<(int)((nwin + 31) / 32), 32, 0, s>>>(
            SincArgs{{kx, ky, kz}, {(int)a.n0, (int)a.n1, (int)a.n2h}, deconv}, win);
        a.wx = win;
        a.wy = win + a.n0;
        a.wz = win + a.n0 + a.n1;
    }
    const size_t sm = nbin <= SMEM_BINS ? 4 * (size_t)nbin * sizeof(double) : 0;
    auto *kern = sm ? zm ? k_powspec<true, true> : k_powspec<true, false>
                    : zm ? k_powspec<false, true> : k_powspec<false, false>;
    allow_smem(kern, sm);
    const int grid = stride_grid((a.n0 / 2 + 1) * (zm ? a.n2h : a.n1 / 2 + 1) * 32, ST, resident(kern, sm));
    kern<<<grid, ST, sm, s>>>(a);
    PMX_LAUNCH_CHECK("k_powspec");
    return own.release();
}

extern "C" int pmx_powspec_bin(const float *F, const float *G, int64_t nbatch,
                               const int64_t grid_shape[3], const double *kx, const double *ky,
                               const double *kz, const double *edges, int32_t nedges,
                               int32_t right, int32_t nbin, double deconv, double *ksum,
                               double *psum, double *nsum, void *stream) {
    return powspec_bin(F, G, nbatch, grid_shape, kx, ky, kz, edges, nedges, right, nbin, deconv,
                       ksum, psum, nsum, stream, false);
}

extern "C" int pmx_powspec_bin_zmajor(const float *F, const float *G, int64_t nbatch,
                                      const int64_t grid_shape[3], const double *kx,
                                      const double *ky, const double *kz, const double *edges,
                                      int32_t nedges, int32_t right, int32_t nbin, double deconv,
                                      double *ksum, double *psum, double *nsum, void *stream) {
    if (grid_shape && (!pow2_grid(grid_shape) || nbin > SMEM_BINS)) {
        clear_error();
        return fail(PMX_ERR_SHAPE, "the (n2h, n0, n1) layout needs a power-of-two grid <= 2048");
    }
    return powspec_bin(F, G, nbatch, grid_shape, kx, ky, kz, edges, nedges, right, nbin, deconv,
                       ksum, psum, nsum, stream, true);
}

extern "C" int pmx_powspec_bin_layout(const float *F, const float *G, int64_t nbatch,
                                      const int64_t grid_shape[3], const double *kx,
                                      const double *ky, const double *kz, const double *edges,
                                      int32_t nedges, int32_t right, int32_t nbin, double deconv,
                                      double *ksum, double *psum, double *nsum, int32_t half_major,
                                      void *scratch, void *stream) {
    return powspec_bin(F, G, nbatch, grid_shape, kx, ky, kz, edges, nedges, right, nbin, deconv,
                       ksum, psum, nsum, stream, half_major != 0, scratch);
}

extern "C" int64_t pmx_powspec_scratch_bytes(const int64_t grid_shape[3], int32_t nedges,
                                             int32_t nbin, int32_t deconv, int32_t sums,
                                             int32_t half_major) {
    if (!grid_shape || nedges < 1 || nbin < 1) return 0;
    for (int a = 0; a < 3; ++a)
        if (grid_shape[a] < 1) return 0;
    return (int64_t)scratch_of(grid_shape, nedges, nbin, deconv != 0, sums != 0, half_major != 0)
        .bytes();
}
