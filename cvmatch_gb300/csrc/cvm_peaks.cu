// cvm_peaks.cu -- every occurrence from a score map, on the device.
//
// The MatchMap recipe of cvmatch_test.go:324-381 (README.md:82-90): a
// result (x, y) is an occurrence when its score is not below the threshold
// and no score within dx in [-rx, rx], dy in [-ry, ry] (clipped to the map)
// is strictly greater.  Occurrences are listed in raster order, so a list
// cut at the caller's capacity keeps the first ones, deterministically.
//
// Three launches: per (row, block of 256 columns) the occurrences' bit mask
// and count; one exclusive scan of the counts in raster order; each block
// writes its occurrences at its scanned offset, ranked by the mask's bits.
//
// Nearly every result is rejected by its score or by one of its eight
// neighbours; what is left is a local maximum, and only those look at their
// whole window.  A warp whose candidates are few takes them one after another,
// its lanes along the window's rows; with many of them (small windows, plateaus
// of equal scores) each lane scans its own.  kLaneScan has the line and its
// figures.
#include "cvm_device.cuh"

namespace cvm {
namespace {

constexpr int kPeakCols = 256;

// A lane's own scan of its window costs the warp one load per window position;
// a candidate taken by the warp one batch of eight loads per eight rows and 32
// columns started, and the batch's latency: as long as kLaneScan positions.
// Measured on 1249 x 769 maps with lines at 8, 16, 32 and 64: 17 x 17 windows
// of noise 89, 82, 65 and 62 us, 33 x 33 of scattered equal peaks 308, 282, 229
// and 261, 81 x 81 of noise 112, 112, 237 and 246.  Every candidate taken by
// the warp: a plateau with 3 x 3 windows 406 us, with 9 x 9 735, 9 x 9 noise 85;
// now 21, 49 and 43.
constexpr int kLaneScan = 32;

// The recipe's test, with its comparisons: a score that is not below the
// threshold (NaN included) is a candidate, and any strictly greater
// neighbour rejects it.  Every lane of the warp takes part.
__device__ __forceinline__ unsigned int peak_bits(const float *__restrict__ m, int w, int h, int x, int y, float thresh,
                                                  int rx, int ry) {
    const int lane = threadIdx.x & 31;
    float v = 0.f;
    bool cand = false;
    if (x < w) {
        v = m[(size_t)y * w + x];
        cand = !(v < thresh);
    }
    if (cand) {
        // the neighbours inside the window and the map, all eight in flight
        // (others stand in as the result itself, which rejects nothing)
        const int xl = rx > 0 ? max(x - 1, 0) : x, xr = rx > 0 ? min(x + 1, w - 1) : x;
        const int yu = ry > 0 ? max(y - 1, 0) : y, yd = ry > 0 ? min(y + 1, h - 1) : y;
        const float *u = m + (size_t)yu * w, *c = m + (size_t)y * w, *d = m + (size_t)yd * w;
        const bool g = (u[xl] > v) | (u[x] > v) | (u[xr] > v) | (c[xl] > v) | (c[xr] > v) | (d[xl] > v) | (d[x] > v) |
                       (d[xr] > v);
        cand = !g;
    }
    unsigned int left = __ballot_sync(0xffffffffu, cand);
    if (rx <= 1 && ry <= 1) return left;  // the neighbours are the window
    const long long batches = (long long)((2 * ry + 8) / 8) * ((2 * rx + 32) / 32);
    if ((2 * rx + 1LL) * (2 * ry + 1) <= kLaneScan * batches * __popc(left)) {
        if (cand) {
            const int x0 = max(0, x - rx), x1 = min(w - 1, x + rx), y0 = max(0, y - ry), y1 = min(h - 1, y + ry);
            // a row at a time, four of up to three columns
            const int step = rx <= 1 ? 4 : 1;
            for (int r = y0; r <= y1 && cand; r += step) {
                bool g = false;
                if (rx <= 1) {
                    for (int c = x0; c <= x1; c++) {
#pragma unroll
                        for (int i = 0; i < 4; i++) g |= m[(size_t)min(r + i, y1) * w + c] > v;
                    }
                } else {
                    const float *row = m + (size_t)r * w;
#pragma unroll 4
                    for (int c = x0; c <= x1; c++) g |= row[c] > v;
                }
                cand = !g;
            }
        }
        return __ballot_sync(0xffffffffu, cand);
    }
    unsigned int bits = 0u;
    for (; left; left &= left - 1) {
        const int l = __ffs(left) - 1, cx = x - lane + l;
        const float cv = __shfl_sync(0xffffffffu, v, l);
        const int x0 = max(0, cx - rx), x1 = min(w - 1, cx + rx), y0 = max(0, y - ry), y1 = min(h - 1, y + ry);
        bool greater = false;
        for (int r = y0; r <= y1 && !greater; r += 8) {
            bool g = false;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float *row = m + (size_t)min(r + i, y1) * w;
                for (int c = x0 + lane; c <= x1; c += 32) g |= row[c] > cv;
            }
            greater = __any_sync(0xffffffffu, g);
        }
        if (!greater) bits |= 1u << l;
    }
    return bits;
}

__global__ void __launch_bounds__(kPeakCols) k_peaks_count(const float *__restrict__ m, int w, int h, float thresh,
                                                            int rx, int ry, int *counts, unsigned int *masks) {
    const int y = blockIdx.y, x = blockIdx.x * kPeakCols + threadIdx.x;
    const unsigned int b = peak_bits(m, w, h, x, y, thresh, rx, ry);
    const size_t block = (size_t)y * gridDim.x + blockIdx.x;
    __shared__ int wc[kPeakCols / 32];
    if ((threadIdx.x & 31) == 0) {
        masks[block * (kPeakCols / 32) + (threadIdx.x >> 5)] = b;
        wc[threadIdx.x >> 5] = __popc(b);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int i = 0; i < kPeakCols / 32; i++) t += wc[i];
        counts[block] = t;
    }
}

// Exclusive scan of n counts in place (one CTA of 1024 threads); the total
// goes to *total.
__global__ void __launch_bounds__(1024) k_peaks_scan(int *counts, int n, int *total) {
    __shared__ int part[1024];
    const int tid = threadIdx.x, per = (n + 1023) / 1024;
    const int a = tid * per, b = min(n, a + per);
    int s = 0;
    for (int i = a; i < b; i++) s += counts[i];
    part[tid] = s;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int v = tid >= o ? part[tid - o] : 0;
        __syncthreads();
        part[tid] += v;
        __syncthreads();
    }
    int run = part[tid] - s;
    for (int i = a; i < b; i++) {
        const int c = counts[i];
        counts[i] = run;
        run += c;
    }
    if (tid == 1023) *total = part[1023];
}

// A thread per 32 results finds their place; the warp writes the words that
// have any one after another, a lane per result.
__global__ void __launch_bounds__(256) k_peaks_write(const int *__restrict__ offsets,
                                                     const unsigned int *__restrict__ masks, int nxb, int words,
                                                     int32_t *xy, int maxPeaks) {
    constexpr int kWords = kPeakCols / 32;
    const int i = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31;
    const unsigned int b = i < words ? masks[i] : 0u;
    const int block = i / kWords, word = i - block * kWords, y = block / nxb;
    const int x = (block - y * nxb) * kPeakCols + 32 * word;
    int idx = 0;
    if (b) {
        idx = offsets[block];
        for (int k = 0; k < word; k++) idx += __popc(masks[block * kWords + k]);
    }
    for (unsigned int left = __ballot_sync(0xffffffffu, b && idx < maxPeaks); left; left &= left - 1) {
        const int l = __ffs(left) - 1;
        const unsigned int bl = __shfl_sync(0xffffffffu, b, l);
        const int at = __shfl_sync(0xffffffffu, idx, l) + __popc(bl & ((1u << lane) - 1u));
        const int xl = __shfl_sync(0xffffffffu, x, l) + lane, yl = __shfl_sync(0xffffffffu, y, l);
        if ((bl >> lane & 1u) && at < maxPeaks) {
            xy[2 * (size_t)at] = xl;
            xy[2 * (size_t)at + 1] = yl;
        }
    }
}

}  // namespace

// a count and the mask's words per block
size_t peaks_scratch_ints(int w, int h) { return (size_t)h * ((w + kPeakCols - 1) / kPeakCols) * (1 + kPeakCols / 32); }

cudaError_t launch_peaks(const float *map, int w, int h, float thresh, int rx, int ry, int *scratch, int32_t *xy,
                         int maxPeaks, int *count, cudaStream_t st) {
    const int nxb = (w + kPeakCols - 1) / kPeakCols;
    const dim3 grid(nxb, h);
    rx = min(rx, w);  // wider windows are the whole row or column
    ry = min(ry, h);
    const size_t blocks = (size_t)nxb * h;
    unsigned int *masks = reinterpret_cast<unsigned int *>(scratch + blocks);
    {
        ProfScope ps("k_peaks_count", st);
        k_peaks_count<<<grid, kPeakCols, 0, st>>>(map, w, h, thresh, rx, ry, scratch, masks);
    }
    {
        ProfScope ps("k_peaks_scan", st);
        k_peaks_scan<<<1, 1024, 0, st>>>(scratch, nxb * h, count);
    }
    if (maxPeaks > 0) {
        ProfScope ps("k_peaks_write", st);
        const int words = (int)(blocks * (kPeakCols / 32));
        k_peaks_write<<<(words + 255) / 256, 256, 0, st>>>(scratch, masks, nxb, words, xy, maxPeaks);
    }
    count_launches(maxPeaks > 0 ? 3 : 2);
    return cudaGetLastError();
}

}  // namespace cvm
