// prep.cu -- per-job set-up kernel: Taylor windows, |k_r| filter and the
// per-pulse geometry table, for every job of a batch in one launch.
//
// A cluster of up to kCluster CTAs per (job, part): part 0 sample window +
// filter (+ clears the job's max|z| and status words), part 1 pulse window,
// part 2 pulse geometry.  What bounds it is the latency of the f64 cosines (a
// term of the window each) and of the maxima over the whole window, so the
// elements are spread over the cluster's threads and the maxima go through
// distributed shared memory: S = 8192 takes 10 us against 64 us with
// one CTA a part, S = 1024 with P = 1999 7 us against 15 us.  In batches of many
// jobs the start of the CTAs is the bound (see launch_prep).
#include <cooperative_groups.h>

#include "internal.h"
#include "kernels.h"

namespace sarbp {

namespace {

constexpr int kPrepThreads = 256, kCluster = 8;
constexpr int kKeep = 4;  // window values a thread keeps between the maximum and the division

namespace cg = cooperative_groups;

// Maxima of N values over a cluster of CL CTAs (fmax: the order does not change them).
template <int CL, int N>
__device__ void cluster_max(double (&v)[N]) {
    __shared__ double part[kPrepThreads / 32][N], mine[N];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = 0; k < N; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] = fmax(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    if (lane == 0)
        for (int k = 0; k < N; ++k) part[warp][k] = v[k];
    __syncthreads();
    if (threadIdx.x < N) {
        double m = part[0][threadIdx.x];
        for (int w = 1; w < kPrepThreads / 32; ++w) m = fmax(m, part[w][threadIdx.x]);
        mine[threadIdx.x] = m;
    }
    if constexpr (CL == 1) {
        __syncthreads();
        for (int k = 0; k < N; ++k) v[k] = mine[k];
    } else {
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        for (int k = 0; k < N; ++k) {
            double m = mine[k];
            for (int r = 0; r < CL; ++r) m = fmax(m, cl.map_shared_rank(mine, r)[k]);
            v[k] = m;
        }
        cl.sync();  // no CTA leaves while another reads its maxima
    }
}

// Taylor window before normalisation, signal.h:43-45:
// w(x) = 1 + sum_r F_m(r) cos(2 pi (r+1) xi), xi = linspace(-0.5, 0.5, num)
__device__ double taylor_w(const DevJob &jb, int num, int x) {
    const double step = (0.5 - (-0.5)) / (double)(num - 1);
    double xi = -0.5 + (double)x * step;
    xi = fmin(fmax(xi, -0.5), 0.5);
    double w = 1.0;
    for (int r = 0; r < jb.n_taylor; ++r)
        w = w + jb.taylor_F[r] * cos((2.0 * 3.14159265358979323846) * (double)(r + 1) * xi);
    return w;
}

// An orthonormal frame (rows of E) for the tiles' window bound: the image
// plane the reference builds by default, u_hat along the ground projection
// of the mid-aperture position, v_hat = z x u_hat, n_hat = z
// (img_plane.cpp:56-75 with n_hat = (0, 0, 1)); the x, y, z axes when that
// projection vanishes.  It depends on the antenna positions only, so the
// r-array and axes forms of a job get the same frame.  Any orthonormal frame
// keeps the bound valid; the image plane's own makes it tight.
__device__ void image_frame(const DevJob &jb, double (&E)[3][3]) {
    for (int i = 0; i < 3; ++i)
        for (int c = 0; c < 3; ++c) E[i][c] = i == c ? 1.0 : 0.0;
    const int m = jb.P / 2;
    double x, y;
    if (jb.precision == SARBP_PREC_PRECISE_ && jb.pos64) {
        x = jb.pos64[3 * m];
        y = jb.pos64[3 * m + 1];
    } else {
        x = jb.pos32[3 * m];
        y = jb.pos32[3 * m + 1];
    }
    const double n = sqrt(x * x + y * y);
    if (!(n > 0.0) || !isfinite(n)) return;
    E[0][0] = x / n;
    E[0][1] = y / n;
    E[0][2] = 0.0;
    E[1][0] = -y / n;
    E[1][1] = x / n;
    E[1][2] = 0.0;
}

template <int CL>
__device__ __forceinline__ void prep_part(const DevJob &jb, int what, int rank) {
    const int first = rank * kPrepThreads + threadIdx.x;  // this thread's first element
    constexpr int kStride = CL * kPrepThreads;
    if (what == 0 || what == 1) {
        const int num = what == 0 ? jb.S : jb.P;
        float *dst = what == 0 ? jb.wS : jb.wP;
        double m[1] = {-INFINITY}, keep[kKeep];
#pragma unroll
        for (int i = 0; i < kKeep; ++i) {
            const int x = first + i * kStride;
            keep[i] = x < num ? taylor_w(jb, num, x) : -INFINITY;
            m[0] = fmax(m[0], keep[i]);
        }
        for (int x = first + kKeep * kStride; x < num; x += kStride) m[0] = fmax(m[0], taylor_w(jb, num, x));
        cluster_max<CL>(m);
#pragma unroll
        for (int i = 0; i < kKeep; ++i) {
            const int x = first + i * kStride;
            if (x < num) dst[x] = (float)(keep[i] / m[0]);
        }
        for (int x = first + kKeep * kStride; x < num; x += kStride) dst[x] = (float)(taylor_w(jb, num, x) / m[0]);
        if (what == 0) {
            for (int s = first; s < jb.S; s += kStride) {
                float f;
                if (jb.precision == SARBP_PREC_PRECISE_ && jb.k_r64)
                    f = (float)fabs(jb.k_r64[s]);
                else
                    f = fabsf(jb.k_r32[s]);
                jb.filt[s] = f;
            }
            if (first == 0) {
                jb.sc->maxabs = 0ull;
                jb.sc->status = 0;
                if (jb.host_status)
                    for (int k = 0; k < kStatusWords; ++k) *reinterpret_cast<volatile int *>(jb.host_status + k) = 0;
                const int h = jb.S / 2;  // k_c = k_r[S/2] (backprojection.cpp:123)
                jb.sc->k_c = (jb.precision == SARBP_PREC_PRECISE_ && jb.k_r64) ? jb.k_r64[h]
                                                                               : (double)jb.k_r32[h];
            }
        }
    } else {
        double E[3][3];
        image_frame(jb, E);
        // maxima of |pos . E_i| / |pos|, and of -|pos|
        double la[4] = {0.0, 0.0, 0.0, -INFINITY};
        for (int p = first; p < jb.P; p += kStride) {
            double4 g;
            if (jb.precision == SARBP_PREC_PRECISE_) {
                double x, y, z;
                if (jb.pos64) {
                    x = jb.pos64[3 * p]; y = jb.pos64[3 * p + 1]; z = jb.pos64[3 * p + 2];
                } else {
                    x = jb.pos32[3 * p]; y = jb.pos32[3 * p + 1]; z = jb.pos32[3 * p + 2];
                }
                double s = __dmul_rn(x, x);
                s = __dadd_rn(s, __dmul_rn(y, y));
                s = __dadd_rn(s, __dmul_rn(z, z));
                g = make_double4(x, y, z, sqrt(s));
            } else {
                // norm_r0 of the reference: f32 (x*x + y*y) + z*z, no fused
                // multiply-add, correctly rounded sqrt (backprojection.cpp:108,
                // util.h:67-71 on the f32 pos buffer).
                const float x = jb.pos32[3 * p], y = jb.pos32[3 * p + 1], z = jb.pos32[3 * p + 2];
                float s = __fmul_rn(x, x);
                s = __fadd_rn(s, __fmul_rn(y, y));
                s = __fadd_rn(s, __fmul_rn(z, z));
                g = make_double4(x, y, z, (double)__fsqrt_rn(s));
            }
            jb.pulse[p] = g;
            const double n = sqrt(g.x * g.x + g.y * g.y + g.z * g.z);
            if (n > 0.0 && isfinite(n)) {
                for (int i = 0; i < 3; ++i)
                    la[i] = fmax(la[i], fabs(g.x * E[i][0] + g.y * E[i][1] + g.z * E[i][2]) / n);
                la[3] = fmax(la[3], -n);
            } else {
                la[3] = 0.0;  // no bound from this job's positions
            }
        }
        cluster_max<CL>(la);
        if (first == 0) {
            for (int i = 0; i < 3; ++i) {
                jb.sc->los_abs[i] = la[i];
                for (int c = 0; c < 3; ++c) jb.sc->frame[i][c] = E[i][c];
            }
            jb.sc->pos_min = -la[3];
        }
    }
}

template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(kPrepThreads)
    prep_cluster_kernel(const DevJob *__restrict__ jobs) {
    prep_part<CL>(jobs[blockIdx.x / CL], blockIdx.y, blockIdx.x % CL);
}
__global__ void __launch_bounds__(kPrepThreads) prep_kernel(const DevJob *__restrict__ jobs) {
    prep_part<1>(jobs[blockIdx.x], blockIdx.y, 0);
}

// The same for one job whose descriptor comes as a kernel parameter, which
// also stores it and makes the job's lists: no upload has to come first (the
// copy and the gaps around it were 15 us of a 256^2 image's 72).
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kPrepThreads)
    prep_single_kernel(const __grid_constant__ DevJob job, const SingleLists l) {
    const int i0 = (blockIdx.y * kCluster + blockIdx.x) * kPrepThreads + threadIdx.x;
    constexpr int kAll = 3 * kCluster * kPrepThreads;
    constexpr int kWords = sizeof(DevJob) / sizeof(uint32_t);
    static_assert(sizeof(DevJob) % sizeof(uint32_t) == 0 && kWords <= kAll, "one word a thread");
    if (i0 < kWords) reinterpret_cast<uint32_t *>(l.job)[i0] = reinterpret_cast<const uint32_t *>(&job)[i0];
    for (int i = i0; i < l.nitems; i += kAll) l.items[i] = WorkItem{0, i % l.ntiles, i / l.ntiles};
    for (int i = i0; i < l.nrows; i += kAll) l.rows[i] = RowItem{0, i};
    for (int i = i0; i < l.ncounters; i += kAll) l.counters[i] = 0;
    prep_part<kCluster>(job, blockIdx.y, blockIdx.x);
}

}  // namespace

// A thread's turn of an element takes about 1.4 us and the start of a CTA of a
// cluster 7 ns of the launch, so of clusters of C CTAs the best C is about the
// root of longest / (4 njobs); each line lies half-way to the next size.  300 jobs of
// 60 x 64: 16 us with one CTA a part, 69 with eight; 96 of 1999 x 1024: 20 with
// two, 37 and 23 with eight and one; 48 of 200 x 8192: 27 with eight, 66 with one.
void launch_prep(const DevJob *d_jobs, int njobs, int longest, cudaStream_t st) {
    auto pays = [&](int c) { return longest > kPrepThreads * c / 2 && 2ll * c * c * njobs <= longest; };
    if (pays(8))
        prep_cluster_kernel<8><<<dim3(njobs * 8, 3), kPrepThreads, 0, st>>>(d_jobs);
    else if (pays(4))
        prep_cluster_kernel<4><<<dim3(njobs * 4, 3), kPrepThreads, 0, st>>>(d_jobs);
    else if (pays(2))
        prep_cluster_kernel<2><<<dim3(njobs * 2, 3), kPrepThreads, 0, st>>>(d_jobs);
    else
        prep_kernel<<<dim3(njobs, 3), kPrepThreads, 0, st>>>(d_jobs);
}

cudaError_t launch_prep_single(const DevJob &job, const SingleLists &lists, cudaStream_t st) {
    prep_single_kernel<<<dim3(kCluster, 3), kPrepThreads, 0, st>>>(job, lists);
    return cudaGetLastError();
}

}  // namespace sarbp
