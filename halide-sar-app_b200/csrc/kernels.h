// kernels.h -- launch wrappers of the device kernels (host-callable).
#pragma once

#include <cuda_runtime.h>

#include "internal.h"
#include "sarbp_b200.h"

#define SARBP_PREC_COMPAT_ SARBP_PREC_COMPAT
#define SARBP_PREC_PRECISE_ SARBP_PREC_PRECISE
#define SARBP_PREC_NAIVE_ SARBP_PREC_NAIVE

namespace sarbp {

// prep.cu
// longest: the most pulses or samples of a job
void launch_prep(const DevJob *d_jobs, int njobs, int longest, cudaStream_t st);
// One job: its descriptor goes to `job`, its work items (part-major: items
// [0, ntiles) are part 0 of each tile, the tile list of the geometry kernels)
// and rows [0, nrows) are listed, and counters[0 .. ncounters) cleared.
struct SingleLists {
    DevJob *job;
    WorkItem *items;
    int ntiles, nitems;
    RowItem *rows;
    int nrows;
    int *counters;
    int ncounters;
};
cudaError_t launch_prep_single(const DevJob &job, const SingleLists &lists, cudaStream_t st);

// range_compress.cu
int twiddle_table_size(int logN);
void fill_twiddle_table(int logN, float2 *host);
cudaError_t launch_range_compress(int logN, const DevJob *d_jobs, const RowItem *d_rows, int nrows, int pairs,
                                  const float2 *d_tw, cudaStream_t st);
cudaError_t init_range_compress_attributes();
// N_fft above 2^kMaxLogNSmem: a four-step FFT through `work`, which holds
// work_rows rows of N_fft complex values (rows go through it work_rows at a
// time; rc_work_rows(logN) rows, rc_work_bytes(logN) bytes, is about
// 256 MB); tw1 and tw2 are the tables of logN / 2 and logN - logN / 2, twN
// the W_N^(n2 k1) table (logN 15..17).
int rc_work_rows(int logN);
size_t rc_work_bytes(int logN);
cudaError_t launch_range_compress_large(int logN, const DevJob *d_jobs, const RowItem *d_rows, int nrows,
                                        int pairs, const float2 *tw1, const float2 *tw2, const float2 *twN,
                                        float2 *work, int work_rows, cudaStream_t st);

// backproject.cu
// Persistent launches: from item `zone` of the list on, an SM takes another
// item only while what it took is below total / SMs, counted in items
// (kDealItems: all equally long; zone and total are set by the launch) or in
// pulses (kDealPulses).
enum { kDealNone = 0, kDealItems = 1, kDealPulses = 2 };
struct BpDeal {
    int how;
    int zone;
    long long total;
};
struct BpLaunch {
    int tile_x, tile_y;
    int minb;        // CTAs per SM the kernel's registers are sized for (2 or 3)
    int stage_cap;   // float4 entries of each half of the staging double buffer
    int cmax;        // max pulses per chunk
    int persistent;  // 1: grid = resident CTAs pulling items from *counter
    int grid;        // CTAs when persistent
    BpDeal deal;     // how a persistent launch shares out the end of its list
    int parts;       // requested pulse parts per tile (sarbp_opts::pulse_parts)
};
bool bp_tile_supported(int tile_x, int tile_y, int minb);
size_t bp_smem_bytes(const BpLaunch &L);
int bp_max_active_blocks(const BpLaunch &L);
cudaError_t init_backproject_attributes();
// d_counter: kBpCounterBytes of device memory (kBpDealBytes with kDealPulses),
// zero before a persistent launch; word kBpZeroWord stays zero
constexpr int kBpZeroWord = 3;
// Most pulse parts that a tile's last item adds itself: it reads them one after
// another, the combine kernel several at once (20 tiles of 118x147 pixels in
// 16 parts replayed: 83 us a plan in place, 64 with the combine kernel; in
// four parts they are equal)
constexpr int kMaxSumParts = 4;
constexpr int kBpCounterBytes = 256, kBpDealSms = 252, kBpDealBytes = 16 + 4 * kBpDealSms;
cudaError_t launch_backproject(const BpLaunch &L, const DevJob *d_jobs, const WorkItem *d_items,
                               int nitems, int *d_counter, cudaStream_t st);
cudaError_t launch_backproject_naive(const DevJob *d_jobs, int job, int nu, int nv, cudaStream_t st);

// geometry.cu
// records = 0: tile table and final phases only (pulse-chunked jobs)
cudaError_t launch_tile_setup(const DevJob *d_jobs, const WorkItem *d_items, int nitems, int tile_pixels,
                              cudaStream_t st, int records = 1);
// per-(tile, pulse) records of one pulse chunk over an existing tile table
cudaError_t launch_tile_records(const DevJob *d_jobs, const WorkItem *d_items, int nitems, cudaStream_t st);


// accum_kernels.cu (pulse-chunked jobs)
// a chunk's descriptor to d_dst, its windows and pulse table gathered into
// job.wP and job.pulse, the backprojection's counters cleared
cudaError_t launch_chunk_setup(const DevJob &job, DevJob *d_dst, const double4 *pulse, const float *wP, int P, int q0,
                               int *counters, cudaStream_t st);
cudaError_t launch_finalize(const DevJob &job, long long npix, int num_sms, cudaStream_t st);
// jobs d_list[0 .. nlist) of d_jobs, formed in pulse parts without sum_parts:
// sum of the parts times the final phase into out (row flip), max |z|
cudaError_t launch_combine_parts(const DevJob *d_jobs, const int *d_list, int nlist, long long max_pixels,
                                 int num_sms, cudaStream_t st);

// resize.cu (the reference's data/resize.py resampling)
struct ResizePlan {
    int elem_bytes;        // 4 (f32) or 8 (f64)
    int nc;                // interleaved components resampled independently
    int rows, cols, orows, ocols;
    double zoom[2];        // input / output extent per axis
    int radius[2];         // Gaussian radius per axis; -1: axis not filtered
    int woff[2];           // offset of each axis's weights w[0..radius] in weights
    const double *weights; // host
    double *d_weights;     // room for them on the device
    void *d_taps;          // (orows + ocols) * 32 bytes of scratch: the zoom's taps per index
};
cudaError_t launch_resize(const ResizePlan &p, const void *in, void *out, void *tmp_a, void *tmp_b,
                          double *bounds, cudaStream_t st, int *launches);

// peaks.cu
cudaError_t measure_peaks(int num_sms, cudaStream_t st, double *ffma_per_s, double *mufu_per_s);

// output.cu
// dB image and u8 image of a complex image, each a pass for max |z|^2 and a pass
// over the pixels (two launches); part: kMaxParts doubles of scratch
constexpr int kMaxParts = 4096;
cudaError_t launch_db(const double2 *img, long long n, double *part, double *dB, cudaStream_t st);
cudaError_t launch_img_u8(const double2 *img, long long n, double *part, uint8_t *u8, double lo, double hi,
                          cudaStream_t st);
cudaError_t launch_u8_from_db(const double *dB, long long n, double dB_min, double dB_max,
                              uint8_t *u8, cudaStream_t st);
// u8 images of every job of a batch that asked for one (uses JobScalars::maxabs):
// `chunks` of kU8Chunk pixels, job i's from DevJob::u8_chunk0 on
cudaError_t launch_batch_u8(const DevJob *d_jobs, int njobs, long long chunks, cudaStream_t st);

}  // namespace sarbp
