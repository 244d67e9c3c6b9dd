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
// whole window, one after another, a warp's lanes along its rows.  (One
// thread per result scanning its window from the corner, in the count and
// again in the write: 90 + 86 us on a 1249 x 769 map with 33 x 33 windows and
// the threshold 0.3; now 30 + 6.)
#include "cvm_device.cuh"

namespace cvm {
namespace {

constexpr int kPeakCols = 256;

// The recipe's test, with its comparisons: a score that is not below the
// threshold (NaN included) is a candidate, and any strictly greater
// neighbour rejects it.  Every lane of the warp takes part.
__device__ __forceinline__ unsigned int peak_bits(const float *__restrict__ m, int w, int h, int x, int y, float thresh,
                                                  int rx, int ry) {
    const int lane = threadIdx.x & 31;
    bool cand = false;
    float v = 0.f;
    if (x < w) {
        const float *p = m + (size_t)y * w + x;
        v = *p;
        cand = !(v < thresh);
        if (cand) {
            const int x0 = rx > 0 && x > 0 ? -1 : 0, x1 = rx > 0 && x + 1 < w ? 1 : 0;
            const int y0 = ry > 0 && y > 0 ? -1 : 0, y1 = ry > 0 && y + 1 < h ? 1 : 0;
            for (int dy = y0; dy <= y1; dy++)
                for (int dx = x0; dx <= x1; dx++) cand = cand && !(p[(long long)dy * w + dx] > v);
        }
    }
    unsigned int bits = 0u;
    for (unsigned int left = __ballot_sync(0xffffffffu, cand); left; left &= left - 1) {
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

// One thread per 32 results.
__global__ void __launch_bounds__(256) k_peaks_write(const int *__restrict__ offsets,
                                                     const unsigned int *__restrict__ masks, int nxb, int words,
                                                     int32_t *xy, int maxPeaks) {
    constexpr int kWords = kPeakCols / 32;
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= words) return;
    unsigned int b = masks[i];
    if (!b) return;
    const int block = i / kWords, word = i - block * kWords, y = block / nxb;
    int idx = offsets[block];
    for (int k = 0; k < word; k++) idx += __popc(masks[block * kWords + k]);
    for (; b && idx < maxPeaks; b &= b - 1, idx++) {
        xy[2 * idx] = (block - y * nxb) * kPeakCols + 32 * word + __ffs(b) - 1;
        xy[2 * idx + 1] = y;
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
