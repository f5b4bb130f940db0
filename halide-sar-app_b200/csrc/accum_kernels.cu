// accum_kernels.cu -- kernels of pulse-chunked image formation (see accum.cpp).
//
// A pulse-chunked job forms its image from consecutive groups of phase-
// history rows.  The descriptor kept on the device is rewritten in stream
// order for each launch (the kernels take it as a parameter, so no host
// synchronisation is needed between chunks); per chunk:
//   chunk_setup_kernel   stores the descriptor, gathers the chunk's pulse
//                        window and pulse table from the whole aperture's
//                        (the reference pairs phase-history row q with
//                        antenna position (q - P mod 2) mod P: the pulse
//                        axis is fftshifted twice, backprojection.cpp:98,104)
//                        and clears the launch counters, in one launch (two
//                        launches and a memset were 10 us of a 200-pulse
//                        chunk's 210 at 1024^2 pixels)
//   range compression, tile records, backprojection (adds to acc)
// and once at the end
//   finalize_kernel      out[nv-1-y][x] = acc[y][x] * fin[y][x]
//                        (backprojection.cpp:130-135), max |z| for dB/u8.
// The combine kernel does the same for one-shot jobs formed in pulse parts
// (each part's sums in its own slice; see DevJob::nsplit).
#include <cstdint>

#include "internal.h"
#include "kernels.h"

namespace sarbp {

namespace {

constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads) chunk_setup_kernel(const __grid_constant__ DevJob job, DevJob *dst,
                                                                const double4 *__restrict__ pulse,
                                                                const float *__restrict__ wP, int P, int q0,
                                                                int *__restrict__ counters) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0) {
        for (int w = threadIdx.x; w < (int)(sizeof(DevJob) / sizeof(uint32_t)); w += kThreads)
            reinterpret_cast<uint32_t *>(dst)[w] = reinterpret_cast<const uint32_t *>(&job)[w];
        if (threadIdx.x < kBpCounterBytes / (int)sizeof(int)) counters[threadIdx.x] = 0;
    }
    if (i >= job.P) return;
    const int q = q0 + i;
    const int p = (q - (P & 1) + P) % P;
    job.wP[i] = wP[q];
    job.pulse[i] = pulse[p];
}

__global__ void __launch_bounds__(kThreads) finalize_kernel(const __grid_constant__ DevJob jb) {
    const long long n = (long long)jb.nu * jb.nv;
    double zmax = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const int iy = (int)(i / jb.nu), ix = (int)(i - (long long)iy * jb.nu);
        const float2 a = jb.acc[i], f = jb.fin[i];
        // the same arithmetic as the backprojection kernel's epilogue
        const double zr = (double)fmaf(a.x, f.x, -a.y * f.y);
        const double zi = (double)fmaf(a.x, f.y, a.y * f.x);
        jb.out[(long long)(jb.nv - 1 - iy) * jb.nu + ix] = make_double2(zr, zi);
        zmax = fmax(zmax, sqrt(zr * zr + zi * zi));
    }
    for (int o = 16; o > 0; o >>= 1) zmax = fmax(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
    __shared__ double s[kThreads / 32];
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = zmax;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kThreads / 32; ++w) zmax = fmax(zmax, s[w]);
        atomicMax(&jb.sc->maxabs, (unsigned long long)__double_as_longlong(zmax));
    }
}

// Jobs formed in pulse parts: out[nv-1-y][x] = (sum of the nsplit slices,
// in slice order) * fin[y][x], the same arithmetic as the backprojection
// kernel's epilogue; max |z| for the u8 image.  blockIdx.y: entry of the job list.
__global__ void __launch_bounds__(kThreads) combine_parts_kernel(const DevJob *__restrict__ jobs,
                                                                 const int *__restrict__ list) {
    const DevJob &jb = jobs[list[blockIdx.y]];
    const long long n = (long long)jb.nu * jb.nv;
    const int ns = jb.nsplit;
    const float2 *__restrict__ parts = jb.parts;
    double zmax = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const int iy = (int)(i / jb.nu), ix = (int)(i - (long long)iy * jb.nu);
        const float2 f = jb.fin[i];
        float2 a = parts[i];
#pragma unroll 4
        for (int k = 1; k < ns; ++k) {
            const float2 b = parts[(long long)k * n + i];
            a.x += b.x;
            a.y += b.y;
        }
        const double zr = (double)fmaf(a.x, f.x, -a.y * f.y);
        const double zi = (double)fmaf(a.x, f.y, a.y * f.x);
        jb.out[(long long)(jb.nv - 1 - iy) * jb.nu + ix] = make_double2(zr, zi);
        if (jb.out_u8) zmax = fmax(zmax, sqrt(zr * zr + zi * zi));
    }
    if (!jb.out_u8) return;
    for (int o = 16; o > 0; o >>= 1) zmax = fmax(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&jb.sc->maxabs, (unsigned long long)__double_as_longlong(zmax));
}

int blocks_for(long long n) {
    long long b = (n + kThreads - 1) / kThreads;
    return (int)(b < 1 ? 1 : b);
}

}  // namespace

cudaError_t launch_chunk_setup(const DevJob &job, DevJob *d_dst, const double4 *pulse, const float *wP, int P, int q0,
                               int *counters, cudaStream_t st) {
    chunk_setup_kernel<<<blocks_for(job.P), kThreads, 0, st>>>(job, d_dst, pulse, wP, P, q0, counters);
    return cudaGetLastError();
}

cudaError_t launch_finalize(const DevJob &job, long long npix, int num_sms, cudaStream_t st) {
    long long b = (npix + kThreads - 1) / kThreads;
    if (b > (long long)num_sms * 8) b = (long long)num_sms * 8;
    finalize_kernel<<<(int)(b < 1 ? 1 : b), kThreads, 0, st>>>(job);
    return cudaGetLastError();
}

cudaError_t launch_combine_parts(const DevJob *d_jobs, const int *d_list, int nlist, long long max_pixels,
                                 int num_sms, cudaStream_t st) {
    if (nlist <= 0) return cudaSuccess;
    long long b = (max_pixels + kThreads - 1) / kThreads;
    const long long cap = ((long long)num_sms * 8 + nlist - 1) / nlist;
    if (b > cap) b = cap;
    combine_parts_kernel<<<dim3((unsigned)(b < 1 ? 1 : b), (unsigned)nlist), kThreads, 0, st>>>(d_jobs, d_list);
    return cudaGetLastError();
}

}  // namespace sarbp
