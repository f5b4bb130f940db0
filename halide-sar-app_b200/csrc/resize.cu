// resize.cu -- resampling of platform arrays on the device: the computation
// the reference's data/resize.py applies to phs, pos and k_r to change the
// pulse and sample counts of a recorded phase history
// (data/resize.py:14-70, `skimage.transform.resize(a, shape,
// preserve_range=True)` with its defaults: linear interpolation, mode
// 'reflect', anti-aliasing when an axis shrinks, output clipped to the input
// range).  scikit-image is not part of the reference (an unpinned
// third-party dependency, absent here); the steps below restate its
// published algorithm (skimage >= 0.19 `resize`, built on scipy.ndimage):
//
//   1. anti-aliasing, on every axis with factor f = in / out > 1: a Gaussian
//      of sigma (f - 1) / 2, truncated at 4 sigma (radius int(4 sigma + 0.5)),
//      weights exp(-x^2 / (2 sigma^2)) normalised to sum 1, applied along
//      axis 0 then axis 1 as a correlation with mirrored edges
//      (x[-k] = x[k], x[n-1+k] = x[n-1-k]), each pass accumulated in f64 as
//      x[i] w0 + sum_{k = r..1} (x[i-k] + x[i+k]) w_k and rounded to the
//      array's type;
//   2. zoom to the output shape, grid-aligned: output index o of an axis
//      samples input coordinate c = (o + 0.5) (in / out) - 0.5, mirrored
//      into [0, n-1]; linear weights (1 - t, t) of the two neighbours
//      floor(c), floor(c) + 1 (mirrored at the edge); the four neighbours of
//      a 2-D sample summed in f64 in row-major order, each value times its
//      axis-0 weight then its axis-1 weight; rounded to the array's type;
//   3. clipped to [min, max] of the unfiltered input.
// One or two components and row filters of radius up to kMaxTileRadius (row
// factors up to 3.9) go through one kernel that takes a tile of the output
// from input to result on chip (resize_tile_kernel); anything else through a
// kernel per step.
// Arrays are [rows][cols][ncomp] of f32 or f64; each of the ncomp
// interleaved components (re, im of a complex array) is resampled on its
// own, as the reference does with np.real and np.imag.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>

#include "internal.h"
#include "kernels.h"

namespace sarbp {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ long long mirror_index(long long m, long long n) {
    if (m >= 0 && m < n) return m;  // inside: no reflection
    if (n <= 1) return 0;
    const long long period = 2 * n - 2;
    if (m < 0) m = -m;
    m %= period;
    return m >= n ? period - m : m;
}

// Launch shape of the per-column kernels: x over the columns of a row, y
// over rows (strided; gridDim.y <= 65535), about 32 blocks per SM in all.
struct RowGrid {
    dim3 grid;
};
inline RowGrid row_grid(long long rows, long long cols) {
    long long gx = (cols + kThreads - 1) / kThreads;
    long long gy = rows;
    const long long target = 148LL * 32;
    if (gx >= target) gy = 1;
    else gy = std::min<long long>(gy, std::max<long long>(1, target / gx));
    gy = std::min<long long>(gy, 65535);
    return RowGrid{dim3((unsigned)std::max<long long>(1, gx), (unsigned)std::max<long long>(1, gy))};
}

// Components per element: NC > 0 fixed at compile time (1, or 2 for the
// real and imaginary parts of a complex array), NC == 0 taken from nc.
template <int NC>
__device__ __forceinline__ int ncomp(int nc) {
    return NC > 0 ? NC : nc;
}

// One correlation pass along `axis` (0: rows, 1: cols) of [rows][cols][nc]
// with symmetric weights w[0..r] (w[0] the centre).  Thread: one column of
// a row (all its components), rows strided over y.
template <typename T, int NC>
__global__ void gauss_pass_kernel(const T *__restrict__ in, T *__restrict__ out, int rows, int cols, int nc_,
                                  int axis, const double *__restrict__ w, int r) {
    const int nc = ncomp<NC>(nc_);
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += gridDim.x * blockDim.x) {
        for (int row = blockIdx.y; row < rows; row += gridDim.y) {
            const int pos = axis == 0 ? row : c, len = axis == 0 ? rows : cols;
            // first value of the element at position m along the axis
            auto base = [&](long long m) -> long long {
                const long long mm = mirror_index(m, len);
                return (axis == 0 ? mm * cols + c : (long long)row * cols + mm) * nc;
            };
            const long long b0 = base(pos);
            T *o = out + ((long long)row * cols + c) * nc;
            if constexpr (NC > 0) {
                // the components side by side, the taps unrolled, so that
                // the loads of several taps are in flight together
                double acc[NC];
#pragma unroll
                for (int k = 0; k < NC; ++k) acc[k] = (double)in[b0 + k] * w[0];
#pragma unroll 4
                for (int t = r; t >= 1; --t) {
                    const long long bm = base((long long)pos - t), bp = base((long long)pos + t);
                    const double wt = w[t];
#pragma unroll
                    for (int k = 0; k < NC; ++k) acc[k] += ((double)in[bm + k] + (double)in[bp + k]) * wt;
                }
#pragma unroll
                for (int k = 0; k < NC; ++k) o[k] = (T)acc[k];
            } else {
                for (int kk = 0; kk < nc; ++kk) {
                    double acc = (double)in[b0 + kk] * w[0];
                    for (int t = r; t >= 1; --t)
                        acc += ((double)in[base((long long)pos - t) + kk] + (double)in[base((long long)pos + t) + kk]) *
                               w[t];
                    o[kk] = (T)acc;
                }
            }
        }
    }
}

// sample coordinate of output index o on an axis of in -> out points
__device__ __forceinline__ double grid_coord(int o, double zoom, long long len) {
    double cc = ((double)o + 0.5) * zoom - 0.5;
    if (len <= 1) return 0.0;
    const double sz2 = (double)(2 * len - 2);
    if (cc < 0) cc = -cc;
    if (cc >= sz2) cc = cc - sz2 * (double)(long long)(cc / sz2);
    if (cc >= (double)len) cc = sz2 - cc;
    return cc;
}

// The two neighbours (mirrored) and linear weights of output index o.
struct Taps {
    long long i0, i1;
    double w0, w1;
};
__device__ __forceinline__ Taps taps_of(int o, double zoom, long long len) {
    const double c = grid_coord(o, zoom, len);
    const double f = floor(c);
    const double t = c - f;
    const long long a = (long long)f;
    return Taps{mirror_index(a, len), mirror_index(a + 1, len), 1.0 - t, t};
}

// taps[0 .. orows) of the output rows, taps[orows .. orows + ocols) of the
// output columns
__global__ void taps_kernel(Taps *__restrict__ taps, int orows, int ocols, double z0, double z1, int rows,
                            int cols) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < orows) taps[i] = taps_of(i, z0, rows);
    else if (i < orows + ocols) taps[i] = taps_of(i - orows, z1, cols);
}

// Thread: one output column (all its components), output rows strided
// over y; the four neighbours summed in f64 in row-major order, each value
// times its row weight then its column weight.
template <typename T, int NC>
__global__ void zoom_kernel(const T *__restrict__ in, T *__restrict__ out, int rows, int cols, int nc_,
                            int orows, int ocols, const Taps *__restrict__ taps, const double *__restrict__ bounds) {
    const int nc = ncomp<NC>(nc_);
    for (int oc = blockIdx.x * blockDim.x + threadIdx.x; oc < ocols; oc += gridDim.x * blockDim.x) {
        const Taps tc = taps[orows + oc];
#pragma unroll 4
        for (int orow = blockIdx.y; orow < orows; orow += gridDim.y) {
            const Taps tr = taps[orow];
            const T *p00 = in + (tr.i0 * cols + tc.i0) * nc, *p01 = in + (tr.i0 * cols + tc.i1) * nc;
            const T *p10 = in + (tr.i1 * cols + tc.i0) * nc, *p11 = in + (tr.i1 * cols + tc.i1) * nc;
            T *o = out + ((long long)orow * ocols + oc) * nc;
#pragma unroll
            for (int k = 0; k < (NC > 0 ? NC : 1); ++k) {
                for (int kk = k; kk < nc; kk += (NC > 0 ? NC : 1)) {
                    double t = 0.0, coeff;
                    coeff = (double)p00[kk];
                    coeff *= tr.w0;
                    coeff *= tc.w0;
                    t += coeff;
                    coeff = (double)p01[kk];
                    coeff *= tr.w0;
                    coeff *= tc.w1;
                    t += coeff;
                    coeff = (double)p10[kk];
                    coeff *= tr.w1;
                    coeff *= tc.w0;
                    t += coeff;
                    coeff = (double)p11[kk];
                    coeff *= tr.w1;
                    coeff *= tc.w1;
                    t += coeff;
                    o[kk] = (T)fmin(fmax(t, bounds[2 * kk]), bounds[2 * kk + 1]);  // the bounds are values of type T
                }
            }
        }
    }
}

// [min, max] of each component: partial bounds of kBoundBlocks slices of
// the array (part[b][k] = (lo, hi)), then one block per component reduces
// them (fmin / fmax: the order does not change the result)
constexpr int kBoundBlocks = 148 * 4;

template <typename T, int NC>
__global__ void __launch_bounds__(kThreads) bounds_partial_kernel(const T *__restrict__ in, long long count, int nc_,
                                                                  double *__restrict__ part) {
    // NC > 0: the NC components in one sweep; NC == 0: one sweep per component
    constexpr int KB = NC > 0 ? NC : 1;
    const int nc = NC > 0 ? NC : nc_;
    __shared__ double slo[KB][kThreads / 32], shi[KB][kThreads / 32];
    for (int k0 = 0; k0 < nc; k0 += KB) {
        double lo[KB], hi[KB];
#pragma unroll
        for (int k = 0; k < KB; ++k) {
            lo[k] = DBL_MAX;
            hi[k] = -DBL_MAX;
        }
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count;
             i += (long long)gridDim.x * blockDim.x) {
#pragma unroll
            for (int k = 0; k < KB; ++k) {
                const double v = (double)in[i * nc + k0 + k];
                lo[k] = fmin(lo[k], v);
                hi[k] = fmax(hi[k], v);
            }
        }
#pragma unroll
        for (int k = 0; k < KB; ++k) {
            for (int o = 16; o > 0; o >>= 1) {
                lo[k] = fmin(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
                hi[k] = fmax(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
            }
            if ((threadIdx.x & 31) == 0) {
                slo[k][threadIdx.x >> 5] = lo[k];
                shi[k][threadIdx.x >> 5] = hi[k];
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll
            for (int k = 0; k < KB; ++k) {
                double l = slo[k][0], h = shi[k][0];
                for (int w = 1; w < kThreads / 32; ++w) {
                    l = fmin(l, slo[k][w]);
                    h = fmax(h, shi[k][w]);
                }
                part[((long long)blockIdx.x * nc + k0 + k) * 2] = l;
                part[((long long)blockIdx.x * nc + k0 + k) * 2 + 1] = h;
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kThreads) bounds_final_kernel(const double *__restrict__ part, int nparts, int nc,
                                                                double *__restrict__ bounds) {
    const int k = blockIdx.x;
    double lo = DBL_MAX, hi = -DBL_MAX;
    for (int b = threadIdx.x; b < nparts; b += blockDim.x) {
        lo = fmin(lo, part[((long long)b * nc + k) * 2]);
        hi = fmax(hi, part[((long long)b * nc + k) * 2 + 1]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __shared__ double slo[kThreads / 32], shi[kThreads / 32];
    if ((threadIdx.x & 31) == 0) {
        slo[threadIdx.x >> 5] = lo;
        shi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kThreads / 32; ++w) {
            lo = fmin(lo, slo[w]);
            hi = fmax(hi, shi[w]);
        }
        bounds[2 * k] = lo;
        bounds[2 * k + 1] = hi;
    }
}

// ---- all steps of one output tile in one kernel ----
// A CTA forms `orn` x `ocn` outputs.  Its input window (the rows and columns
// that the tile's neighbours and their filters touch, mirrored at the edges)
// is read once, a thread to a column running down the rows with the row
// filter's 2 R0 + 1 values in registers; the filtered rows go to shared
// memory, where the column filter and the linear weights are applied per
// output.  The clip bounds need the whole input, so the CTAs collect the
// extremes of what they read and of what they wrote, and clip_kernel goes over
// the output only if something lies outside (values rounded past the extremes,
// NaN).  The filters' sums are written as the roundings of the step kernels'
// loops (left to the compiler, the unrolled row filter merged the centre's
// product instead of the first pair's, and values differed in the last place),
// so both paths give the same values bit for bit.  A kernel per step moved the array through memory four times: 1999 x
// 1800 complex128 to half 129 us, 59 us in one; to twice 129 -> 81
// us; 2000 x 2000 to a quarter 192 -> 75 us.
constexpr int kMaxTileRadius = 6;          // of the row filter
constexpr int kMaxTileColRadius = 15;      // of the column filter
constexpr int kTileCols = 128;            // window columns, 256 / kTileCols row segments
constexpr size_t kTileSmem = 48 * 1024;   // filtered rows
constexpr int kMaxTileRows = 64, kMaxTileCols = 256;  // outputs of a tile
constexpr int kMinTileRows = 4, kTileSplit = 148;      // (see tile_shape)

// Extremes of a component as bits that order like the values, all from 0 on:
// [0] ~min in, [1] max in, [2] ~min out, [3] max out, [4] NaN written.
constexpr int kStatWords = 5;
__device__ __forceinline__ unsigned long long ordered_bits(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : b | (1ull << 63);
}
__device__ __forceinline__ double from_ordered(unsigned long long o) {
    return __longlong_as_double((long long)((o >> 63) ? o & ~(1ull << 63) : ~o));
}

// the filters' weights, as a kernel parameter (no upload comes first)
struct TileWeights {
    double w0[kMaxTileRadius + 1], w1[kMaxTileColRadius + 1];
};

struct TileTap {
    int i0, i1;  // neighbours, then relative to the window
    double t;    // weight of i1; 1 - t of i0
};

// the extremes with NaN left out, as fmin and fmax (b NaN: a)
template <typename T>
__device__ __forceinline__ T min_of(T a, T b) { return b < a ? b : a; }
template <typename T>
__device__ __forceinline__ T max_of(T a, T b) { return b > a ? b : a; }

template <typename T, int NC>
struct __align__(sizeof(T) * NC) Elem {
    T v[NC];
};

// R0: radius of the row filter, -1 without; r1 likewise of the column filter.
template <typename T, int NC, int R0>
__global__ void __launch_bounds__(256, 3)
    resize_tile_kernel(const T *__restrict__ in_, T *__restrict__ out_, int rows, int cols, int orows, int ocols,
                       double z0, double z1, const __grid_constant__ TileWeights w, int r1, int orn, int ocn,
                       unsigned long long *__restrict__ stats) {
    using E = Elem<T, NC>;
    const E *in = reinterpret_cast<const E *>(in_);
    E *out = reinterpret_cast<E *>(out_);
    extern __shared__ __align__(16) unsigned char smem[];
    E *win = reinterpret_cast<E *>(smem);
    __shared__ int lim[4];  // first and last window row and column
    const int tid = threadIdx.x;
    const int tiles_c = (ocols + ocn - 1) / ocn;
    const int or0 = (blockIdx.x / tiles_c) * orn, oc0 = (blockIdx.x % tiles_c) * ocn;
    const int nr = min(orn, orows - or0), nc = min(ocn, ocols - oc0);
    TileTap *taps = reinterpret_cast<TileTap *>(smem + kTileSmem);  // rows, then columns
    if (tid < 4) lim[tid] = (tid & 1) ? -1 : 0x7fffffff;
    __syncthreads();
    for (int i = tid; i < nr + nc; i += 256) {
        const bool row = i < nr;
        const Taps t = row ? taps_of(or0 + i, z0, rows) : taps_of(oc0 + i - nr, z1, cols);
        taps[i] = TileTap{(int)t.i0, (int)t.i1, t.w1};
        atomicMin(&lim[row ? 0 : 2], (int)min(t.i0, t.i1));
        atomicMax(&lim[row ? 1 : 3], (int)max(t.i0, t.i1));
    }
    __syncthreads();
    const int r1h = max(r1, 0);
    const int lo = lim[0], nrow = lim[1] - lo + 1, clo = lim[2], ncol = lim[3] - clo + 1 + 2 * r1h;
    // an extreme that no value has taken: f64's largest, rounded to T
    constexpr T kNone = sizeof(T) == 4 ? (T)INFINITY : (T)DBL_MAX;
    T ilo[NC], ihi[NC], olo[NC], ohi[NC];
    int nan = 0;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        ilo[k] = olo[k] = kNone;
        ihi[k] = ohi[k] = -kNone;
    }
    // ---- row filter, down the rows of a segment of the window ----
    {
        constexpr int kSegs = 256 / kTileCols, RH = R0 > 0 ? R0 : 0, RING = 2 * RH + 1;
        const int c = tid % kTileCols, seg = tid / kTileCols;
        const int a = nrow * seg / kSegs, b = nrow * (seg + 1) / kSegs;
        if (c < ncol && a < b) {
            const E *col = in + mirror_index(clo - r1h + c, cols);
            double wt[RH + 1];
#pragma unroll
            for (int t = 0; t <= RH; ++t) wt[t] = R0 >= 0 ? w.w0[t] : 1.0;
            E ring[RING];
            const bool inside = lo - RH >= 0 && lo + nrow + RH <= rows;
            const E *p = col + (long long)(lo + a - RH) * cols;  // where inside
            auto load = [&](int row) {
                E e;
                if (inside) {
                    e = *p;
                    p += cols;
                } else {
                    e = col[mirror_index(row, rows) * cols];
                }
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    ilo[k] = min_of(ilo[k], e.v[k]);
                    ihi[k] = max_of(ihi[k], e.v[k]);
                }
                return e;
            };
#pragma unroll
            for (int j = 0; j < RING - 1; ++j) ring[j + 1] = load(lo + a - RH + j);
            E *dst = win + a * ncol + c;
#pragma unroll 4
            for (int i = a; i < b; ++i, dst += ncol) {
#pragma unroll
                for (int j = 0; j < RING - 1; ++j) ring[j] = ring[j + 1];
                ring[RING - 1] = load(lo + i + RH);
                E f = ring[RH];
                if (R0 >= 0) {
#pragma unroll
                    for (int k = 0; k < NC; ++k) {
                        double acc = __dmul_rn((double)ring[RH].v[k], wt[0]);
#pragma unroll
                        for (int t = RH; t >= 1; --t)
                            acc = __fma_rn((double)ring[RH - t].v[k] + (double)ring[RH + t].v[k], wt[t], acc);
                        f.v[k] = (T)acc;
                    }
                }
                *dst = f;
            }
        }
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    // ---- column filter in place, a warp to a row ----
    if (r1 >= 0) {
        constexpr int kSteps = kTileCols / 32;
        for (int i = warp; i < nrow; i += 8) {
            E *row = win + i * ncol + r1h;
            E f[kSteps];
#pragma unroll
            for (int q = 0; q < kSteps; ++q) {
                const int c = lane + 32 * q;
                if (c < ncol - 2 * r1h) {
                    double acc[NC];
#pragma unroll
                    for (int k = 0; k < NC; ++k) acc[k] = __dmul_rn((double)row[c].v[k], w.w1[0]);
                    for (int t = r1; t >= 1; --t) {
                        const E m = row[c - t], n = row[c + t];
                        const double wt = w.w1[t];
#pragma unroll
                        for (int k = 0; k < NC; ++k) acc[k] = __fma_rn((double)m.v[k] + (double)n.v[k], wt, acc[k]);
                    }
#pragma unroll
                    for (int k = 0; k < NC; ++k) f[q].v[k] = (T)acc[k];
                }
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < kSteps; ++q)
                if (lane + 32 * q < ncol - 2 * r1h) row[lane + 32 * q] = f[q];
        }
        __syncthreads();
    }
    // ---- linear weights, an output at a time ----
    for (int c = lane; c < nc; c += 32) {
        const TileTap tc = taps[nr + c];
        const double c0 = 1.0 - tc.t;
        for (int r = warp; r < nr; r += 8) {
            const TileTap tr = taps[r];
            const double r0 = 1.0 - tr.t;
            const E *q0 = win + (tr.i0 - lo) * ncol + r1h - clo, *q1 = win + (tr.i1 - lo) * ncol + r1h - clo;
            const E p00 = q0[tc.i0], p01 = q0[tc.i1], p10 = q1[tc.i0], p11 = q1[tc.i1];
            E o;
#pragma unroll
            for (int k = 0; k < NC; ++k) {
                double t = 0.0, coeff;
                coeff = (double)p00.v[k];
                coeff *= r0;
                coeff *= c0;
                t += coeff;
                coeff = (double)p01.v[k];
                coeff *= r0;
                coeff *= tc.t;
                t += coeff;
                coeff = (double)p10.v[k];
                coeff *= tr.t;
                coeff *= c0;
                t += coeff;
                coeff = (double)p11.v[k];
                coeff *= tr.t;
                coeff *= tc.t;
                t += coeff;
                o.v[k] = (T)t;  // rounding is monotonic: it may come before the clip
                olo[k] = min_of(olo[k], o.v[k]);
                ohi[k] = max_of(ohi[k], o.v[k]);
                nan |= t != t;
            }
            out[(long long)(or0 + r) * ocols + oc0 + c] = o;
        }
    }
    // ---- extremes ----
#pragma unroll
    for (int k = 0; k < NC; ++k)
        for (int s = 16; s > 0; s >>= 1) {
            ilo[k] = min_of(ilo[k], __shfl_xor_sync(0xffffffffu, ilo[k], s));
            ihi[k] = max_of(ihi[k], __shfl_xor_sync(0xffffffffu, ihi[k], s));
            olo[k] = min_of(olo[k], __shfl_xor_sync(0xffffffffu, olo[k], s));
            ohi[k] = max_of(ohi[k], __shfl_xor_sync(0xffffffffu, ohi[k], s));
        }
    nan = __syncthreads_or(nan);  // and the window is no longer read
    double *red = reinterpret_cast<double *>(smem);
    if ((tid & 31) == 0)
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            double *d = red + ((tid >> 5) * NC + k) * 4;
            d[0] = ilo[k];
            d[1] = ihi[k];
            d[2] = olo[k];
            d[3] = ohi[k];
        }
    __syncthreads();
    if (tid < 4 * NC) {
        const int k = tid >> 2, what = tid & 3;
        double m = red[k * 4 + what];
        for (int w = 1; w < 8; ++w) {
            const double v = red[(w * NC + k) * 4 + what];
            m = (what & 1) ? fmax(m, v) : fmin(m, v);
        }
        atomicMax(&stats[k * kStatWords + what], (what & 1) ? ordered_bits(m) : ~ordered_bits(m));
        if (nan && what == 0) atomicMax(&stats[k * kStatWords + 4], 1ull);
    }
}

// Clips the output to the extremes of the input where it exceeds them.
template <typename T, int NC>
__global__ void __launch_bounds__(256) clip_kernel(T *__restrict__ out, long long count,
                                                   const unsigned long long *__restrict__ stats) {
    double lo[NC], hi[NC];
    bool any = false;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const unsigned long long *s = stats + k * kStatWords;
        lo[k] = from_ordered(~s[0]);
        hi[k] = from_ordered(s[1]);
        any = any || s[4] || from_ordered(~s[2]) < lo[k] || from_ordered(s[3]) > hi[k];
    }
    if (!any) return;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < count; i += 256LL * gridDim.x)
#pragma unroll
        for (int k = 0; k < NC; ++k) out[i * NC + k] = (T)fmin(fmax((double)out[i * NC + k], lo[k]), hi[k]);
}

// Tile shape of a plan: false where the tile kernel does not apply (it reads
// whole elements, and the output may not lie over the input).
template <typename T>
bool tile_shape(const ResizePlan &p, const void *in, const void *out, int *orn, int *ocn) {
    if ((p.nc != 1 && p.nc != 2) || p.radius[0] > kMaxTileRadius || p.radius[1] > kMaxTileColRadius) return false;
    const uintptr_t i0 = reinterpret_cast<uintptr_t>(in), o0 = reinterpret_cast<uintptr_t>(out);
    const size_t elem = p.nc * sizeof(T);
    if (i0 % elem || o0 % elem) return false;
    if (i0 < o0 + (size_t)p.orows * p.ocols * elem && o0 < i0 + (size_t)p.rows * p.cols * elem) return false;
    // an axis of zoom z takes at most z (n - 1) + 3 window positions for n outputs
    const int r1 = std::max(p.radius[1], 0);
    const double c = (kTileCols - 3 - 2 * r1) / p.zoom[1];
    if (c < 8.0) return false;
    *ocn = (int)std::min<double>({c, (double)kMaxTileCols, (double)p.ocols});
    const double wcols = std::min<double>(kTileCols, std::ceil(p.zoom[1] * *ocn) + 3 + 2 * r1);
    const double r = std::floor((double)kTileSmem / (wcols * p.nc * sizeof(T))) - 3;
    if (r < p.zoom[0]) return false;
    *orn = (int)std::min<double>({r / p.zoom[0], (double)kMaxTileRows, (double)p.orows});
    if (*orn < 1) return false;
    auto ctas = [&] { return (long long)((p.orows + *orn - 1) / *orn) * ((p.ocols + *ocn - 1) / *ocn); };
    // fewer rows a tile where SMs would have no tile (64^2 complex128 to 64 x
    // 1000: 20.6 us in 4 tiles of 64 rows, 12.4 in 64 of 4; the steps 16.5)
    while (*orn > kMinTileRows && ctas() < kTileSplit) *orn = (*orn + 1) / 2;
    // A few long rows leave most of a CTA idle, and its fixed cost (3.5 us a
    // round of 444) is more than the steps' in many rounds, where the steps have
    // no filter to run above all (f64, tiles and steps: 1 x 1000000 to 400000 70
    // us and 38, 4 x 250000 to half 31 and 43; 2 x 1000000 to 3 x 1000000 64 and
    // 48, 2 x 350000 to 3 x 350000 29 and 32, 7 x 700000 complex to 8 rows 86 and 88)
    const long long n = std::max(p.rows, p.orows), bytes = n * (long long)elem;
    if (p.radius[0] < 0 && p.radius[1] < 0) return n > 8 || bytes > 100 || ctas() <= (n > 1 ? 3300 : 2000);
    return n > 6 || bytes > 48 || ctas() <= 1000 * (n + 1);
}

template <typename T, int NC>
cudaError_t launch_tiles(const ResizePlan &p, const T *in, T *out, unsigned long long *stats, int orn, int ocn,
                         cudaStream_t st) {
    const long long tiles = (long long)((p.orows + orn - 1) / orn) * ((p.ocols + ocn - 1) / ocn);
    // The kernel's limit belongs to the device, not to a context, so every call
    // sets it to the most that any tile needs: a call's own size would refuse
    // the launch of another thread's larger tile that comes just after it
    constexpr int kSmemLimit = (int)(kTileSmem + (kMaxTileRows + kMaxTileCols) * sizeof(TileTap));
    const size_t smem = kTileSmem + (size_t)(orn + ocn) * sizeof(TileTap);
    cudaError_t e = cudaMemsetAsync(stats, 0, NC * kStatWords * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    TileWeights w{};
    for (int t = 0; t <= p.radius[0]; ++t) w.w0[t] = p.weights[p.woff[0] + t];
    for (int t = 0; t <= p.radius[1]; ++t) w.w1[t] = p.weights[p.woff[1] + t];
    switch (p.radius[0]) {
#define X(R)                                                                                                        \
    case R:                                                                                                         \
        e = cudaFuncSetAttribute(resize_tile_kernel<T, NC, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit); \
        if (e != cudaSuccess) return e;                                                                             \
        resize_tile_kernel<T, NC, R><<<(unsigned)tiles, 256, smem, st>>>(in, out, p.rows, p.cols, p.orows, p.ocols,  \
                                                                         p.zoom[0], p.zoom[1], w, p.radius[1], orn,  \
                                                                         ocn, stats);                               \
        break;
        X(-1) X(0) X(1) X(2) X(3) X(4) X(5) X(6)
#undef X
        default: return cudaErrorInvalidValue;
    }
    const long long count = (long long)p.orows * p.ocols;
    const long long b = std::max<long long>(1, std::min<long long>((count + 1023) / 1024, 148 * 4));
    clip_kernel<T, NC><<<(unsigned)b, 256, 0, st>>>(out, count, stats);
    return cudaGetLastError();
}

template <typename T>
cudaError_t resize_t(const ResizePlan &p, const void *in, void *out, void *tmp_a, void *tmp_b, double *bounds,
                     cudaStream_t st, int *launches) {
    const T *src = static_cast<const T *>(in);
    int orn = 0, ocn = 0;
    if (tile_shape<T>(p, in, out, &orn, &ocn)) {
        *launches = 2;
        auto *stats = reinterpret_cast<unsigned long long *>(bounds);
        return p.nc == 1 ? launch_tiles<T, 1>(p, src, static_cast<T *>(out), stats, orn, ocn, st)
                         : launch_tiles<T, 2>(p, src, static_cast<T *>(out), stats, orn, ocn, st);
    }
    *launches = 4 + (p.radius[0] >= 0) + (p.radius[1] >= 0);
    if (p.radius[0] >= 0 || p.radius[1] >= 0) {
        const size_t nw = (size_t)std::max(p.radius[0] >= 0 ? p.woff[0] + p.radius[0] + 1 : 0,
                                           p.radius[1] >= 0 ? p.woff[1] + p.radius[1] + 1 : 0);
        cudaError_t e = cudaMemcpyAsync(p.d_weights, p.weights, nw * sizeof(double), cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return e;
    }
    T *a = static_cast<T *>(tmp_a), *b = static_cast<T *>(tmp_b);
    // bounds[0 .. 2 nc) the result, bounds + 2 nc the partials
    const long long count = (long long)p.rows * p.cols;
    const int nparts = (int)std::min<long long>(kBoundBlocks, (count + kThreads - 1) / kThreads);
    if (p.nc == 1)
        bounds_partial_kernel<T, 1><<<nparts, kThreads, 0, st>>>(src, count, 1, bounds + 2);
    else if (p.nc == 2)
        bounds_partial_kernel<T, 2><<<nparts, kThreads, 0, st>>>(src, count, 2, bounds + 4);
    else
        bounds_partial_kernel<T, 0><<<nparts, kThreads, 0, st>>>(src, count, p.nc, bounds + 2 * p.nc);
    bounds_final_kernel<<<p.nc, kThreads, 0, st>>>(bounds + 2 * p.nc, nparts, p.nc, bounds);
    // anti-aliasing passes, axis 0 then axis 1
    const T *cur = src;
    for (int axis = 0; axis < 2; ++axis) {
        if (p.radius[axis] < 0) continue;
        T *dst = (cur == a) ? b : a;
        const dim3 g = row_grid(p.rows, p.cols).grid;
        const double *w = p.d_weights + p.woff[axis];
        if (p.nc == 1)
            gauss_pass_kernel<T, 1><<<g, kThreads, 0, st>>>(cur, dst, p.rows, p.cols, 1, axis, w, p.radius[axis]);
        else if (p.nc == 2)
            gauss_pass_kernel<T, 2><<<g, kThreads, 0, st>>>(cur, dst, p.rows, p.cols, 2, axis, w, p.radius[axis]);
        else
            gauss_pass_kernel<T, 0><<<g, kThreads, 0, st>>>(cur, dst, p.rows, p.cols, p.nc, axis, w, p.radius[axis]);
        cur = dst;
    }
    Taps *taps = static_cast<Taps *>(p.d_taps);
    const int ntaps = p.orows + p.ocols;
    taps_kernel<<<(ntaps + kThreads - 1) / kThreads, kThreads, 0, st>>>(taps, p.orows, p.ocols, p.zoom[0],
                                                                       p.zoom[1], p.rows, p.cols);
    const dim3 g = row_grid(p.orows, p.ocols).grid;
    T *o = static_cast<T *>(out);
    if (p.nc == 1)
        zoom_kernel<T, 1><<<g, kThreads, 0, st>>>(cur, o, p.rows, p.cols, 1, p.orows, p.ocols, taps, bounds);
    else if (p.nc == 2)
        zoom_kernel<T, 2><<<g, kThreads, 0, st>>>(cur, o, p.rows, p.cols, 2, p.orows, p.ocols, taps, bounds);
    else
        zoom_kernel<T, 0><<<g, kThreads, 0, st>>>(cur, o, p.rows, p.cols, p.nc, p.orows, p.ocols, taps, bounds);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_resize(const ResizePlan &p, const void *in, void *out, void *tmp_a, void *tmp_b,
                          double *bounds, cudaStream_t st, int *launches) {
    if (p.elem_bytes == 4) return resize_t<float>(p, in, out, tmp_a, tmp_b, bounds, st, launches);
    if (p.elem_bytes == 8) return resize_t<double>(p, in, out, tmp_a, tmp_b, bounds, st, launches);
    return cudaErrorInvalidValue;
}

}  // namespace sarbp
