// output.cu -- dB and u8 output stages (img_output.cpp:10-52).
//
//   m   = max |z| over the image               (img_output.cpp:23-24)
//   dB  = 10 * log(|z| / m) / log(10)          (img_output.cpp:26, util.h:56-58;
//         log(Expr(10)) has an integer argument, so Halide takes it in f32)
//   u8  = trunc(clamp((clamp(dB, lo, hi) - lo) / (hi - lo) * 255, 0, 255))
//                                              (img_output.cpp:48-51, signal.h:55-57)
// HBM-bound but for the f64 logarithm of the dB image; the u8 form reads the
// complex image once and writes the u8 image, using the max|z| that the
// backprojection epilogue already reduced where there is one.
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "internal.h"
#include "kernels.h"

namespace sarbp {

namespace {

constexpr double kLn10F32 = 2.302585124969482421875;  // logf(10.0f)

__device__ __forceinline__ uint8_t to_u8(double v, double lo, double hi) {
    if (v != v) v = lo;
    v = fmin(fmax(v, lo), hi);
    double n = (v - lo) / (hi - lo) * 255.0;
    n = fmin(fmax(n, 0.0), 255.0);
    return (uint8_t)n;
}

// u8 of one pixel.  The value is decided in f32 (|z|^2 rounded to f32, the
// accurate logf), whose error is far below 1e-4 of a grey level for display
// ranges of 0.1 dB and wider; a pixel whose f32 level lands within that
// margin of an integer or of the clamps, or whose |z|^2 or ratio to the
// maximum's is not a normal f32 number (below -190 dB), is recomputed with the
// reference's f64 formula.  Pixels clearly
// below dB_min or above dB_max are decided in f32 as well: in a scene of a few
// bright points that is most of them (12 jobs of 256^2 to 1024^2 pixels, -40
// dB: 81 us with those in f64, 31 us without).
struct U8Scale {
    double m, lo, hi;
    float inv_m2, k, q0, eps;  // q = k ln(|z|^2 / m^2) + q0 (grey levels)
};

__device__ __forceinline__ U8Scale u8_scale(double m, double lo, double hi) {
    U8Scale u;
    u.m = m;
    u.lo = lo;
    u.hi = hi;
    const double g = 255.0 / (hi - lo);               // grey levels per dB
    u.inv_m2 = (float)(1.0 / (m * m));
    u.k = (float)(5.0 / kLn10F32 * g);                // 10 log10(a/m) = 5 ln(a^2/m^2) / ln 10
    u.q0 = (float)(-lo * g);
    u.eps = (float)(2e-5 * g + 1e-4);
    if (!(u.inv_m2 >= FLT_MIN && u.inv_m2 <= FLT_MAX)) u.eps = INFINITY;  // every pixel in f64
    return u;
}

__device__ __forceinline__ uint8_t u8_of(double2 z, const U8Scale &u) {
    const double a2 = z.x * z.x + z.y * z.y;
    const float a = (float)a2, x = a * u.inv_m2;
    const float q = fmaf(u.k, logf(x), u.q0);
    const float f = q - floorf(q);
    // an f32 underflow says nothing (nothing overflows: |z| <= m, and m^2 is
    // at most 1 / FLT_MIN unless eps is infinite)
    if (a >= FLT_MIN && x >= FLT_MIN) {
        if (q > u.eps && q < 255.0f - u.eps && f > u.eps && f < 1.0f - u.eps) return (uint8_t)q;
        if (q < -u.eps) return 0;
        if (q > 255.0f + u.eps) return 255;
    }
    return to_u8(10.0 * (log(sqrt(a2) / u.m) / kLn10F32), u.lo, u.hi);
}

// max |z|: four independent 16-byte loads in flight per thread and step (a
// warp's loads stay contiguous), the maximum taken on |z|^2 and one square
// root at the end -- the same value, as the square root is monotonic and
// correctly rounded.
// One maximum of |z|^2 per CTA; the kernel that uses it takes the maximum of
// those (image_max2), so nothing has to be cleared ahead of the pass.
__global__ void __launch_bounds__(256) max2_kernel(const double2 *__restrict__ img, long long n,
                                                   double *__restrict__ part) {
    double m2 = 0.0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * stride < n; i += 4 * stride) {
        double2 z[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) z[k] = img[i + k * stride];
#pragma unroll
        for (int k = 0; k < 4; ++k) m2 = fmax(m2, z[k].x * z[k].x + z[k].y * z[k].y);
    }
    for (; i < n; i += stride) {
        const double2 z = img[i];
        m2 = fmax(m2, z.x * z.x + z.y * z.y);
    }
    for (int o = 16; o > 0; o >>= 1) m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
    __shared__ double s[8];
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = m2;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) m2 = fmax(m2, s[w]);
        part[blockIdx.x] = m2;
    }
}

// Maximum over a warp of values from 0 on, whose bits order as they do.
__device__ __forceinline__ double warp_max_bits(double v) {
    const uint32_t hi = (uint32_t)__double2hiint(v), top = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t lo = __reduce_max_sync(0xffffffffu, hi == top ? (uint32_t)__double2loint(v) : 0u);
    return __hiloint2double((int)top, (int)lo);
}

// max |z|^2 of the image from its partial maxima, in every thread of a CTA of 256
__device__ __forceinline__ double image_max2(const double *__restrict__ part, int nparts) {
    double m2 = 0.0;
    // independent loads: one after another they are several L2 latencies ahead
    // of the first pixel
    for (int i0 = threadIdx.x; i0 < nparts; i0 += 8 * 256) {
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = i0 + 256 * k < nparts ? part[i0 + 256 * k] : 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) m2 = fmax(m2, v[k]);
    }
    m2 = warp_max_bits(m2);
    __shared__ double s[8];
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = m2;
    __syncthreads();
    return warp_max_bits(s[threadIdx.x & 7]);
}

// dB of one pixel.  The reference's 10 (log(|z| / m) / ln 10) takes a square
// root and two divisions besides the logarithm, and the f64 pipe is what
// bounds the kernel; here it is 5 / ln 10 times the logarithm of
// |z|^2 * (1 / m^2).  The factor is held in two parts (24 bits and the rest),
// so that one rounding follows the logarithm where the formula has two: with
// the factor rounded to one f64 every pixel carried that rounding, and the
// error against 80-bit values was 9.3e-16 (rms, 1500 x 1100 speckle)
// against the formula's 7.0e-16; now it is 5.7e-16.  The maximum itself stays
// at exactly 0 and nothing above it; a maximum whose square is not an ordinary
// number, and a pixel whose ratio to it is none (below -1538 dB), takes the
// reference's formula.  2048^2: 22 us, 31 with the formula.
constexpr double kDbHi = (double)(float)(5.0 / kLn10F32);
constexpr double kDbLo = (5.0 - kDbHi * kLn10F32) / kLn10F32;  // (the product is exact: 24 + 24 bits)
static_assert(kDbLo > 0.0, "the parts of -inf (a zero pixel) add up to -inf");
struct DbScale {
    double m2, inv, m;
    bool plain;
};
__device__ __forceinline__ DbScale db_scale(double m2) {
    return DbScale{m2, 1.0 / m2, sqrt(m2), m2 > 1e-290 && m2 < 1e290};
}
__device__ __forceinline__ double db_of(double2 z, const DbScale &s) {
    const double a2 = z.x * z.x + z.y * z.y;
    double q = a2 * s.inv;
    const int hi = __double2hiint(q);  // (range tests on the integer side: the f64 pipe is the busy one)
    if (!s.plain || (hi < 0x00100000 && a2 > 0.0)) return 10.0 * (log(sqrt(a2) / s.m) / kLn10F32);
    if (hi >= 0x3fefffff && (a2 >= s.m2 || q > 1.0)) q = 1.0;
    const double l = log(q);
    return fma(l, kDbHi, l * kDbLo);
}

// Two neighbouring pixels a thread and step: 32 B in, 16 B out where dB is
// 16-byte aligned.
__global__ void __launch_bounds__(256) db_kernel(const double2 *__restrict__ img, long long n,
                                                 const double *__restrict__ part, int nparts,
                                                 double *__restrict__ dB) {
    const DbScale s = db_scale(image_max2(part, nparts));
    const bool vec = (reinterpret_cast<uintptr_t>(dB) & 15) == 0;
    const long long stride = 2LL * gridDim.x * blockDim.x;
    for (long long i = 2 * ((long long)blockIdx.x * blockDim.x + threadIdx.x); i < n; i += stride) {
        if (i + 1 < n) {
            const double2 z0 = img[i], z1 = img[i + 1];
            const double d0 = db_of(z0, s), d1 = db_of(z1, s);
            if (vec) {
                *reinterpret_cast<double2 *>(dB + i) = make_double2(d0, d1);
            } else {
                dB[i] = d0;
                dB[i + 1] = d1;
            }
        } else {
            dB[i] = db_of(img[i], s);
        }
    }
}

__global__ void u8_from_db_kernel(const double *__restrict__ dB, long long n, double lo, double hi,
                                  uint8_t *__restrict__ u8) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        u8[i] = to_u8(dB[i], lo, hi);
}

// u8 of the four neighbouring pixels [i0, i0 + 4) of an image of n pixels:
// 64 B of complex f64 in, one 32-bit word of u8 out when the destination is
// 4-byte aligned (vec).
__device__ __forceinline__ void u8_quad(const double2 *__restrict__ img, long long n, long long i0,
                                        uint8_t *__restrict__ u8, bool vec, const U8Scale &us) {
    if (vec && i0 + 4 <= n) {
        double2 z[4];  // the four loads first, then the conversions
#pragma unroll
        for (int k = 0; k < 4; ++k) z[k] = img[i0 + k];
        uint32_t w = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) w |= (uint32_t)u8_of(z[k], us) << (8 * k);
        *reinterpret_cast<uint32_t *>(u8 + i0) = w;
    } else {
        for (long long i = i0; i < n && i < i0 + 4; ++i) u8[i] = u8_of(img[i], us);
    }
}

// The u8 images of a batch in chunks of kU8Chunk pixels, a job's chunks from
// jb.u8_chunk0 on; each CTA takes a run of chunks, whichever jobs they fall
// into (a fixed number of CTAs per job left the largest images of a mix to
// few: 12 jobs of 256^2 to 1024^2 pixels 92 -> 81 us).  Each thread converts
// four neighbouring pixels.
__global__ void __launch_bounds__(256) batch_u8_kernel(const DevJob *__restrict__ jobs, int njobs, long long total,
                                                       long long per) {
    const long long c0 = blockIdx.x * per, c1 = c0 + per < total ? c0 + per : total;
    int cur = -1;
    U8Scale us;
    for (long long c = c0; c < c1; ++c) {
        // the last job that starts at or before chunk c (jobs without an u8
        // image have no chunks)
        int before = 0;
        for (int j0 = 0; j0 < njobs; j0 += 256) {
            const int j = j0 + (int)threadIdx.x;
            before += __syncthreads_count(j < njobs && jobs[j].u8_chunk0 <= c);
        }
        const DevJob &jb = jobs[before - 1];
        if (cur != before - 1) {
            cur = before - 1;
            us = u8_scale(__longlong_as_double((long long)jb.sc->maxabs), jb.dB_min, jb.dB_max);
        }
        const long long n = (long long)jb.nu * jb.nv, i0 = (c - jb.u8_chunk0) * kU8Chunk + 4 * threadIdx.x;
        if (i0 < n) u8_quad(jb.out, n, i0, jb.out_u8, (reinterpret_cast<uintptr_t>(jb.out_u8) & 3) == 0, us);
    }
}

// The same conversion for one image given by its pointer and the partial
// maxima of max2_kernel.
__global__ void __launch_bounds__(256) img_u8_kernel(const double2 *__restrict__ img, long long n,
                                                     const double *__restrict__ part, int nparts,
                                                     uint8_t *__restrict__ u8, double lo, double hi) {
    const U8Scale us = u8_scale(sqrt(image_max2(part, nparts)), lo, hi);
    const bool vec = ((reinterpret_cast<uintptr_t>(u8) & 3) == 0);
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; 4 * q < n; q += stride)
        u8_quad(img, n, 4 * q, u8, vec, us);
}

int grid_for(long long n) {
    long long b = (n + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    if (b < 1) b = 1;
    return (int)b;
}

// CTAs of 256 threads that the device holds at once for `kernel` (one wave
// of a grid-stride loop: no partial last wave); looked up once per kernel.
template <typename K>
long long resident_ctas(K kernel, int *cache) {
    if (*cache > 0) return *cache;
    int dev = 0, sms = 148, occ = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 256, 0) != cudaSuccess || occ < 1) occ = 4;
    *cache = occ * sms;
    return *cache;
}
int g_max2_ctas = 0, g_img_u8_ctas = 0, g_batch_u8_ctas = 0, g_db_ctas = 0;

// the partial maxima of an image; their number
int launch_max2(const double2 *img, long long n, double *part, cudaStream_t st) {
    // at least eight pixels a thread (two steps of four loads), at most one
    // wave of resident CTAs
    const long long b = std::max<long long>(
        1, std::min<long long>({(n + 2047) / 2048, resident_ctas(max2_kernel, &g_max2_ctas), (long long)kMaxParts}));
    max2_kernel<<<(unsigned)b, 256, 0, st>>>(img, n, part);
    return (int)b;
}

}  // namespace

cudaError_t launch_db(const double2 *img, long long n, double *part, double *dB, cudaStream_t st) {
    const int np = launch_max2(img, n, part, st);
    const long long b = std::max<long long>(1, std::min<long long>((n + 511) / 512, resident_ctas(db_kernel, &g_db_ctas)));
    db_kernel<<<(unsigned)b, 256, 0, st>>>(img, n, part, np, dB);
    return cudaGetLastError();
}

cudaError_t launch_u8_from_db(const double *dB, long long n, double lo, double hi, uint8_t *u8,
                              cudaStream_t st) {
    u8_from_db_kernel<<<grid_for(n), 256, 0, st>>>(dB, n, lo, hi, u8);
    return cudaGetLastError();
}

cudaError_t launch_img_u8(const double2 *img, long long n, double *part, uint8_t *u8, double lo, double hi,
                          cudaStream_t st) {
    const int np = launch_max2(img, n, part, st);
    // one wave of resident CTAs, four pixels per thread and step
    const long long bx = std::max<long long>(
        1, std::min<long long>((n / 4 + 255) / 256, resident_ctas(img_u8_kernel, &g_img_u8_ctas)));
    img_u8_kernel<<<(unsigned)bx, 256, 0, st>>>(img, n, part, np, u8, lo, hi);
    return cudaGetLastError();
}

cudaError_t launch_batch_u8(const DevJob *d_jobs, int njobs, long long chunks, cudaStream_t st) {
    if (chunks <= 0) return cudaSuccess;
    // at most one wave of resident CTAs over the whole batch
    const long long cap = resident_ctas(batch_u8_kernel, &g_batch_u8_ctas);
    const long long per = (chunks + cap - 1) / cap;
    batch_u8_kernel<<<(unsigned)((chunks + per - 1) / per), 256, 0, st>>>(d_jobs, njobs, chunks, per);
    return cudaGetLastError();
}

}  // namespace sarbp
