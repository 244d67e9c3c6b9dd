// cvm_lines.cu -- the inverse row transforms of 2^7 .. 2^11 points, one
// small group of threads per row pair.
//
// inverseRowPair (impl.go:394-444), the channel sum, the correlation's end
// of normOne (impl.go:825-849) and the first-occurrence extrema, with the
// butterflies, twiddles and rounded operations of k_inv_rows_t
// (cvm_rows.cu) in the same order: the scores are the same bits.  What
// differs is who does what.
//
// What bounds it.  A transform of N points is N/16 units of 16 elements per
// pass, so N/16 threads hold a whole line in registers and its passes need
// no more threads than that.  With 256-thread CTAs over several lines (four
// per SM) every pass ended in a barrier over all of them, and the loads of
// the spectrum rows and of the score's denominators (both from DRAM)
// stalled the whole CTA; a third of the 4100 warp instructions per
// 1024-point line were the score ladder of results that are no extremum.
// Here a line belongs to N/16 threads of a 64-thread CTA (128 for N = 2048):
// barriers span two warps (one for N <= 512), the groups drift apart, the
// next row pair's rows and den are on their way to L2 while the current one
// is transformed, and results that cannot be extrema skip the ladder (Track,
// below): 2400 warp instructions per line, 54 % of the issue slots, the
// instructions' own latency first among the stalls.
//
// Measured (GB300, the rows of one FindAll in sequence): 256 RGBA templates
// on 2560x1440, fast form, 571 thousand 1024-point lines: 3.17 -> 1.86 ms;
// 64 templates on 1920x1080, exact form: 1.19 -> 0.83 ms.
//
// Data path of a line: pass 1 combines Z = U + iV (and its mirror) from the
// two spectrum rows on the way into registers, so the combined line is never
// stored; its outputs go to the line buffer; the last pass's outputs are
// scored in registers.  Staging the rows in shared memory (cp.async) instead
// of reading each value twice from L1 measured 2.62 ms: 17 KB per line
// leaves the twiddles no L1.
//
// (Line buffer: cvm_lines.cuh.)
#include "cvm_lines.cuh"

namespace cvm {
namespace {

// Floats as unsigned integers of the same order (every finite float's key is
// above 0, which stands for "none yet").
__device__ __forceinline__ unsigned int ordered_key(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u >> 31) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_key(unsigned int k) {
    return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k);
}

// Only the extrema leave a match without a score map, so a result that
// cannot be one needs no quotient: scores outside (lo, hi) may be extrema.
// hi lies below the largest known score by 2^-20 of it and 1e-15: num < hi *
// den then implies that the computed quotient (within 2 ulp, 2^-22; near-flat
// windows' within half of one) is below that score, the product's rounding
// included (2^-24: a den is 0 or above 1e-6, since idiff / area exceeds its
// guard), and, scores being at most 1 (+ 2 ulp), that num < den.  lo is its
// mirror.  A result at or above the cut, ties included, takes the whole
// ladder.
__device__ __forceinline__ float below(float v) { return v - (fabsf(v) * 9.5367431640625e-07f + 1e-15f); }
__device__ __forceinline__ float above(float v) { return v + (fabsf(v) * 9.5367431640625e-07f + 1e-15f); }

struct Track {
    float minV, maxV, hi, lo;
    int minL, maxL;       // CTA-local raster index (row x N + x)
};

__device__ __forceinline__ void track(Track &t, float sc, int l) {
    if (sc < t.minV || (sc == t.minV && l < t.minL)) {
        t.minV = sc;
        t.minL = l;
    }
    if (sc > t.maxV || (sc == t.maxV && l < t.maxL)) {
        t.maxV = sc;
        t.maxL = l;
    }
}

// A result that may be an extremum.  Out of line: rare, and inlined copies
// of it at sixteen to thirty-two results cost the kernel its instruction
// cache (half its stalls).
template <bool FAST>
__device__ __noinline__ Track score_track(Track t, float num, float den, float denFlat, int l) {
    const float sc = FAST ? score_fast(num, den, denFlat) : score_exact(num, den);
    track(t, sc, l);
    t.hi = fmaxf(t.hi, below(sc));
    t.lo = fminf(t.lo, above(sc));
    return t;
}

// The group's extrema so far as the cuts of all its threads.
__device__ __forceinline__ void cut_share(Track &t, unsigned int mask) {
    const float hi = from_key(__reduce_max_sync(mask, ordered_key(t.maxV)));
    const float lo = -from_key(__reduce_max_sync(mask, ordered_key(-t.minV)));
    if (hi > -FLT_MAX) t.hi = fmaxf(t.hi, below(hi));
    if (lo < FLT_MAX) t.lo = fminf(t.lo, above(lo));
}

// The cuts from the extrema (keys of the maximum and of the negated minimum)
// of the member's CTAs that have finished; false when there are none.
__device__ __forceinline__ bool cut_keys(Track &t, unsigned int kx, unsigned int kn) {
    if (kx) t.hi = fmaxf(t.hi, below(from_key(kx)));
    if (kn) t.lo = fminf(t.lo, above(-from_key(kn)));
    return kx != 0u && kn != 0u;
}

// den and (t, den): read once, so they leave the L1 lines to the twiddles.
__device__ __forceinline__ float ld_once(const float *p) {
    float v;
    asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 ld_once(const float2 *p) {
    float2 v;
    asm("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}


constexpr int kBlocksMax = 1024;  // of a CTA: 8192 results over two rows a pair, in 4 x 4 blocks

// A tallied call's counter in shared memory, behind the blocks' bounds.
template <int L>
__device__ __forceinline__ unsigned int *tally_word() {
    extern __shared__ __align__(16) float2 smem[];
    return reinterpret_cast<unsigned int *>(reinterpret_cast<float *>(smem + (size_t)Lines<L>::NL * Lines<L>::LINE) +
                                            kBlocksMax);
}

// A result above its block's bound: its den, and the ladder unless that
// already rules it out.  (TALLY: the row length of a tallied call, else 0.)
template <int TALLY>
__device__ __noinline__ Track score_table(Track t, float num, const MemberSet &ms, const DevMember &m,
                                          const DevParams &Pm, int y, int x, float denFlat, int l) {
    if constexpr (TALLY > 0) {
        // (the warp's lanes that are here, once)
        const unsigned int here = __activemask();
        if ((threadIdx.x & 31) == __ffs(here) - 1) atomicAdd(tally_word<TALLY>(), 1u);
    }
    const float d = sat_den(ms, m, Pm, y, x);
    if (d > 0.f && num < t.hi * d && num > t.lo * d) return t;
    const float sc = score_fast(num, d, denFlat);
    track(t, sc, l);
    t.hi = fmaxf(t.hi, below(sc));
    t.lo = fminf(t.lo, above(sc));
    return t;
}


// CTAs per SM the registers are budgeted for: 96 registers hold a fast-form
// thread's 32 den values ahead of the last pass (12 CTAs spill: 2.13 against
// 2.01 ms; without them 14 CTAs 2.00 at the same 4096 elements per CTA); the
// exact form keeps the channel sum of its 16 results, 128 registers (nine
// CTAs spill: 1.17 against 0.84 ms).  With every score (mode 0) the quotients
// of all results are in flight too.  Score maps at every length, us with 3, 5,
// 6, 7 and 8 CTAs, RGB in the exact form and gray in the fast form:
//    128  320x200, 16x16       exact 17.8 19.2 18.4 19.9 20.0  fast 14.3 14.3 14.4 14.7 14.4
//    256  1280x800, 32x32      exact 27.6 26.6 23.7 25.6 24.8  fast 16.8 16.5 16.7 17.0 16.7
//    512  1366x767, 133x71     exact 34.3 28.8 25.0 28.6 28.7  fast 26.8 19.1 19.4 19.9 19.4
//    512  2560x1440, 100x60    exact 86.2 92.8 81.1 81.0 81.4  fast 64.6 57.2 56.8 50.3 48.7
//   1024  1920x1080, 96x32     exact 43.4 53.6 49.4 38.0 37.2  fast 26.5 26.8 26.8 20.6 20.2
//   1024  2560x1440, 128x128   exact 73.9 74.4 69.0 63.5 65.3  fast 45.2 39.4 39.4 34.4 34.9
//   2048  3840x2160, 256x256   exact 94.4 134.9 170 170 170    fast 56.9 46.1 47.7 46.8 46.0
__host__ __device__ constexpr int lines_ctas(int L, bool fast, int mode) {
    return mode == 2 || mode == 4 ? (L == 11 ? 4 : (L <= 8 ? 8 : 9))
           : mode == 0            ? (fast ? (L == 11 ? 5 : 7) : (L == 7 || L == 11 ? 3 : (L == 10 ? 7 : 6)))
                                  : (L == 11 ? (fast ? 5 : 4) : (L <= 8 ? (fast ? 10 : 5) : (fast ? 10 : 8)));
}

// What a launch keeps of its results.  ALL: every score is wanted (a score
// map).  LANES: the extrema alone, den (and t)
// from the statistics kernel's lanes.  TABLE: a fast-form fleet's extrema,
// den on demand.  SOLO: LANES for a single match, whose CTAs all start at once
// with no extrema of earlier ones to cut by (fleets keep their registers).
// TALLY: TABLE in a tallied call (MemberSet::formed; the test for it alone, in
// TABLE's registers, cost the rows 4 %).  ROI: LANES for members with regions of
// interest, whose results outside are no candidates and whose row pairs outside
// are not transformed.  (40 gray members on 1280x720, a quarter of the frame
// each: 254.8 us a call; 393 with every score kept and all results of a CTA that
// holds any of the region scored.)
enum Keep { ALL, LANES, TABLE, SOLO, TALLY, ROI };

// The extrema (and scores) of the CTA's row pairs.
template <int L, bool FAST, Keep KEEP>
__device__ __forceinline__ Ext line_pairs(const InvArgs &a, float2 *smem, const DevMember &m, const DevParams &Pm,
                                          const TileBox &tb, int bw, int bh, int pair0, int P, unsigned int *bnd) {
    using S = Lines<L>;
    constexpr Keep MODE = KEEP == TALLY ? TABLE : KEEP;
    constexpr bool LEAN = MODE != ALL;
    constexpr int N = S::N, R1 = S::R1, K1 = S::K1, NB = S::NB, G = S::G, NL = S::NL, PITCH = S::PITCH;
    constexpr int NU = NB == 1 ? 1 : 16 / NB;             // last-pass units of a thread
    constexpr int RL = NB == 1 ? 16 : NB;                 // their radix
    constexpr int HL = NB == 1 ? S::H2 : S::H3;           // their quarter
    constexpr bool BOTH = RL == 4;                        // both rows' den values in registers at once
    constexpr bool AHEAD = BOTH && FAST && MODE != TABLE;  // and every unit's
    const FftClass &fc = a.fc;
    const int slot = blockIdx.x, tileLocal = blockIdx.z, tid = threadIdx.x;
    Ext e;
    const int g = tid / G, lt = tid - g * G;          // the thread's group and its place in it
    const unsigned int mask = G >= 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << ((tid & 31) / G * G);
    float2 *ln = smem + (size_t)g * S::LINE;
    const int hwp = fc.hwp, log2H = fc.log2H;
    const int cn = FAST ? 1 : Pm.cn;
    const size_t chanStride = (size_t)fc.dftH * hwp;
    const float2 *scr = a.ms.scratch[a.cls] + (size_t)slot * a.ms.scratchStride[a.cls] +
                        (size_t)tileLocal * a.cnS * chanStride;
    const float2 *lanes = a.ms.lanes + (size_t)slot * a.ms.lanesStride;
    const float *dens = reinterpret_cast<const float *>(lanes);
    const float denFlat = near_flat_den(m.tw, m.th, Pm.templNorm);  // fast form: near-flat windows below it
    float *map = LEAN ? nullptr : a.ms.map;
    const int rw = m.rw, roiY0 = m.roiY0, roiY1 = m.roiY1;
    // the columns that may be extrema
    const int xa = MODE == ROI ? max(m.roiX0 - tb.x0, 0) : 0, xb = MODE == ROI ? min(m.roiX1 - tb.x0, bw) : bw;
    const float2 *triW = fc.triW;
    int j2, b2;
    pass2_unit<L>(lt, j2, b2);
    bool warm = false;                                // the cuts have been shared once
    float postV = -FLT_MAX, postN = FLT_MAX;          // TABLE: the extrema the warp has posted
    float *lbs = reinterpret_cast<float *>(smem + (size_t)NL * S::LINE);
    int lgx = 0, lgy = 0, nbx = 0;
    if constexpr (MODE == TABLE) {
        lgx = block_log2(m.tw);
        lgy = block_log2(m.th);
        nbx = (bw + (1 << lgx) - 1) >> lgx;
        const int rows = min(2 * P, bh - 2 * pair0), n = nbx * ((rows + (1 << lgy) - 1) >> lgy);
        bool flat = true;
        if (KEEP == TALLY && tid == 0) *tally_word<L>() = 0u;
#pragma unroll 1
        for (int i = tid; i < n; i += S::CTA) {
            const int by = i / nbx, x = (i - by * nbx) << lgx, y = by << lgy;
            const float lb = block_bound(a.ms, m, Pm, tb.y0 + 2 * pair0 + y, tb.x0 + x, min(1 << lgx, bw - x),
                                         min(1 << lgy, rows - y));
            lbs[i] = lb;
            flat = flat && lb == INFINITY;
        }
        // No deviation in any window of the CTA (a black frame, a letterbox's
        // bars): every den and so every score is 0, whatever the correlation.
        // 64 templates on a black 1920x1080 frame: 1.81 ms with the
        // transforms, 0.62 without; with den from the statistics kernel 1.32.
        if (__syncthreads_and(flat)) {
            ext_init(e);
            if (tid == 0) ext_add(e, 0.f, (long long)(tb.y0 + 2 * pair0) * m.rw + tb.x0);
            return e;
        }
    }
    Track t = {FLT_MAX, -FLT_MAX, -INFINITY, INFINITY, INT_MAX, INT_MAX};
    // rows r and r + 1 of channel k
    auto row_ptr = [&](int p, int k, int h) {
        return scr + (size_t)k * chanStride + (size_t)brev_bits(2 * (pair0 + p) + h, log2H) * hwp;
    };
    // towards L2, one 128-byte line per thread and step: the two rows
    // and (last channel) their den
    auto prefetch = [&](int p, int k) {
        for (int o = lt; o < 2 * (N / 32 + 1); o += G) {
            const int h = o > N / 32, c = h ? o - (N / 32 + 1) : o;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(row_ptr(p, k, h) + 16 * c));
        }
        if (MODE != TABLE && k == cn - 1) {
            constexpr int EB = FAST ? 4 : 8;
            const int r = 2 * (pair0 + p);
            for (int h = 0; h < 2 && r + h < bh; h++) {
                const char *q = reinterpret_cast<const char *>(lanes) +
                                ((long long)(tb.y0 + r + h) * rw + tb.x0) * EB;
                for (int o = lt * 128; o < bw * EB; o += G * 128)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(q + o));
            }
        }
    };
    float2 acc[FAST ? 1 : 16];                        // the earlier channels' sum, the thread's results
    for (int p = g; p < P; p += NL) {
        if (MODE == ROI && (tb.y0 + 2 * (pair0 + p) + 2 <= roiY0 || tb.y0 + 2 * (pair0 + p) >= roiY1)) continue;
#pragma unroll 1
        for (int k = 0; k < cn; k++) {
            // pass 1: unit k0's elements are Z[k0 + K1 * brev(i)]
            // (bit-reversed input), Z = U + iV below N/2 and its mirror
            // above (impl.go:405-413)
            const float2 *ur = row_ptr(p, k, 0), *vr = row_ptr(p, k, 1);
            // the member's extrema so far, used at the line's end
            const bool posted = LEAN && bnd && k == cn - 1 && (MODE == TABLE || MODE == ROI || p < NL);
            uint2 keys = make_uint2(0u, 0u);
            if (posted) {
                keys.x = *reinterpret_cast<const volatile unsigned int *>(bnd);
                keys.y = *reinterpret_cast<const volatile unsigned int *>(bnd + 1);
            }
#pragma unroll
            for (int q = 0; q < 16 / R1; q++) {
                const int k0 = lt + q * G;
                float2 z[R1];
                constexpr int LR1 = R1 == 16 ? 4 : 3;
#pragma unroll
                for (int i = 0; i < R1 / 2; i++) {
                    const float2 u = __ldg(ur + k0 + K1 * i), v = __ldg(vr + k0 + K1 * i);
                    z[brevk(i, LR1)] = make_float2(__fsub_rn(u.x, v.y), __fadd_rn(u.y, v.x));
                }
#pragma unroll
                for (int i = R1 / 2; i < R1; i++) {
                    const int n = K1 * (R1 - i) - k0;
                    const float2 u = __ldg(ur + n);
                    float2 v = __ldg(vr + n);
                    float uy = u.y;
                    if (i == R1 / 2 && k0 == 0) {  // N/2 itself: the direct form
                        uy = -uy;
                        v.y = -v.y;
                    }
                    z[brevk(i, LR1)] = make_float2(__fadd_rn(u.x, v.y), __fsub_rn(v.x, uy));
                }
                if constexpr (R1 == 16)
                    math16<true, 1, FAST>(z, triW);
                else
                    math_head<true, FAST>(z, triW);
                // the previous pair's last pass has read the line
                if (q == 0) group_sync<G>(mask);
#pragma unroll
                for (int i = 0; i < R1; i++) ln[i * PITCH + k0] = z[i];
            }
            if (k + 1 < cn || p + NL < P) prefetch(k + 1 < cn ? p : p + NL, k + 1 < cn ? k + 1 : 0);
            group_sync<G>(mask);
            const bool last = k == cn - 1;
            const bool odd = 2 * (pair0 + p) + 1 < bh;  // the imaginary part's row exists
            const int y0 = tb.y0 + 2 * (pair0 + p);
            const long long row0 = (long long)y0 * rw + tb.x0;
            const int blockRow = MODE == TABLE ? ((2 * p) >> lgy) * nbx : 0;  // of both rows
            // den (and t) of the thread's results, unit it
            float den[AHEAD ? NU : 1][BOTH ? 2 : 1][RL], tt[BOTH ? 2 : 1][FAST ? 1 : RL];
            auto load_den = [&](int it, int h) {
                const int jj = lt + it * G, is = AHEAD ? it : 0, hs = BOTH ? h : 0;
                const long long row = row0 + h * rw;
                const int xe = h == 0 || odd ? xb : 0;
#pragma unroll
                for (int i = 0; i < RL; i++) {
                    const int x = jj + HL * i;
                    if constexpr (MODE == TABLE) {
                        den[is][hs][i] = lbs[blockRow + (min(x, bw - 1) >> lgx)];  // its bound
                    } else {
                        float2 td = make_float2(0.f, 0.f);
                        const bool in = x < xe && (MODE != ROI || x >= xa);
                        if constexpr (FAST)
                            td.y = in ? ld_once(dens + row + x) : 0.f;
                        else if (in)
                            td = ld_once(lanes + row + x);
                        if constexpr (!FAST) tt[hs][i] = td.x;
                        den[is][hs][i] = td.y;
                    }
                }
            };
            float2 z[16];
            pass2<L, true, FAST>(ln, j2, b2, z, triW);
            if constexpr (AHEAD) {
                // every unit's, in flight together while the barrier gathers the line
#pragma unroll
                for (int it = 0; it < NU; it++) {
                    load_den(it, 0);
                    load_den(it, 1);
                }
            }
            // `warm` gates collectives of the group's lanes, and other CTAs
            // post while the lanes read: one answer for all of them
            if (LEAN && last && posted) warm = __all_sync(mask, cut_keys(t, keys.x, keys.y)) || warm;
            if constexpr (NB > 1) group_sync<G>(mask);
#pragma unroll
            for (int it = 0; it < NU; it++) {
                // last-pass unit jj: results x = jj + HL * i of the two rows
                const int jj = lt + it * G;
                if (last && !AHEAD) {
                    load_den(it, 0);
                    if (BOTH && MODE != TABLE) load_den(it, 1);
                }
                float2 *o = z;
                float2 zu[NB == 1 ? 1 : RL];
                if constexpr (NB > 1) {
                    pass3<L, true, FAST>(ln, jj, zu, triW);
                    o = zu;
                }
                if (!FAST && !last) {
                    // the channels' sum, in channel order (impl.go:425-443)
#pragma unroll
                    for (int i = 0; i < RL; i++) {
                        float2 &s = acc[FAST ? 0 : it * RL + i];
                        s = k == 0 ? o[i] : make_float2(__fadd_rn(s.x, o[i].x), __fadd_rn(s.y, o[i].y));
                    }
                    continue;
                }
                // the correlation of result i of row h, the earlier channels' sum
                // and t applied (the exact form)
                auto numer = [&](int h, int i) {
                    float num = h ? o[i].y : o[i].x;
                    if constexpr (!FAST) {
                        const float2 s = acc[it * RL + i];
                        if (cn > 1) num = __fadd_rn(h ? s.y : s.x, num);
                        num = __fsub_rn(num, tt[BOTH ? h : 0][i]);
                    }
                    return num;
                };
                if (MODE == SOLO && it == 0 && !warm) {
                    // No extrema to start from (a single match's CTAs all start
                    // at once): the largest and smallest quotients of the warp's
                    // first unit, by the hardware division, as cuts -- within
                    // 2^-22 of scores that are there, cut at 2^-18.  (Without
                    // them nearly all its results took the ladder, 2000 of the
                    // 2500 instructions of a 128-point line's warp.)
                    float qx = -FLT_MAX, qn = FLT_MAX;
#pragma unroll
                    for (int h = 0; h < (BOTH ? 2 : 1); h++)
#pragma unroll
                        for (int i = 0; i < RL; i++) {
                            const float num = numer(h, i), d = den[AHEAD ? it : 0][BOTH ? h : 0][i];
                            const float q = __fdividef(num, d);
                            if (jj + HL * i < bw && fabsf(num) < d) {
                                qx = fmaxf(qx, q);
                                qn = fminf(qn, q);
                            }
                        }
                    qx = from_key(__reduce_max_sync(mask, ordered_key(qx)));
                    qn = -from_key(__reduce_max_sync(mask, ordered_key(-qn)));
                    if (qx > -FLT_MAX) t.hi = fmaxf(t.hi, qx - (fabsf(qx) * 3.814697265625e-06f + 1e-15f));
                    if (qn < FLT_MAX) t.lo = fminf(t.lo, qn + (fabsf(qn) * 3.814697265625e-06f + 1e-15f));
                    warm = true;
                }
                // cuts on either side of 0, or none: a lower bound of den needs
                // them so, and a zero den is then the score 0 between them
                const float hp = t.hi > 0.f ? t.hi : -INFINITY, lp = t.lo < 0.f ? t.lo : INFINITY;
                const float zero = MODE != TABLE && t.hi > 0.f && t.lo < 0.f ? 0.f : -1.f;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if (h == 1 && !odd) break;
                    if (h == 1 && !BOTH && MODE != TABLE) load_den(it, 1);
                    if (MODE == ROI && (y0 + h < roiY0 || y0 + h >= roiY1)) continue;
#pragma unroll
                    for (int i = 0; i < RL; i++) {
                        const int x = jj + HL * i, l = (2 * p + h) * N + x;
                        const float num = numer(h, i);
                        const float d = den[AHEAD ? it : 0][BOTH && MODE != TABLE ? h : 0][i];
                        const bool cand = x < xb && (MODE != ROI || x >= xa) && d != zero &&
                                          !(num < hp * d && num > lp * d);
                        if constexpr (MODE == TABLE) {
                            if (cand)
                                t = score_table<KEEP == TALLY ? L : 0>(t, num, a.ms, m, Pm, y0 + h, tb.x0 + x, denFlat, l);
                        } else if constexpr (LEAN) {
                            if (cand) t = score_track<FAST>(t, num, d, denFlat, l);
                        } else if (x < bw) {
                            const float sc = FAST ? score_fast(num, d, denFlat) : score_exact(num, d);
                            map[row0 + h * rw + x] = sc;
                            track(t, sc, l);
                        }
                    }
                }
                if (LEAN && MODE != SOLO && it == 0 && !warm) {
                    cut_share(t, mask);
                    warm = true;
                }
            }
            // new extrema at once to the member's other CTAs: without a
            // cut every result forms its den
            if (MODE == TABLE && __any_sync(mask, t.maxV > postV || t.minV < postN)) {
                const unsigned int kx = __reduce_max_sync(mask, ordered_key(t.maxV));
                const unsigned int kn = __reduce_max_sync(mask, ordered_key(-t.minV));
                postV = from_key(kx);
                postN = -from_key(kn);
                t.hi = fmaxf(t.hi, below(postV));
                t.lo = fminf(t.lo, above(postN));
                if ((lt & 31) == 0) {
                    atomicMax(bnd, kx);
                    atomicMax(bnd + 1, kn);
                }
            }
        }
    }
    // widen: CTA-local (row, x) -> the member's raster index
    auto widen = [&](int l) {
        return l == INT_MAX ? LLONG_MAX
                            : (long long)(tb.y0 + 2 * pair0 + (l >> L)) * m.rw + tb.x0 + (l & (N - 1));
    };
    e.minV = t.minV;
    e.maxV = t.maxV;
    e.minI = widen(t.minL);
    e.maxI = widen(t.maxL);
    return e;
}

template <int L, bool FAST, Keep MODE>
__global__ void __launch_bounds__(Lines<L>::CTA, lines_ctas(L, FAST, MODE)) k_inv_lines(const __grid_constant__ InvArgs a) {
    griddep_wait();
    using S = Lines<L>;
    extern __shared__ __align__(16) float2 smem[];
    __shared__ Ext shExt[S::CTA / 32];
    __shared__ int isLast;
    const FftClass &fc = a.fc;
    // members vary fastest: a member's CTAs spread over the whole launch, so
    // all but its first start from the extrema of earlier ones (a.bounds)
    const int slot = blockIdx.x, tileLocal = blockIdx.z;
    const int tile = fc.tileFirst + tileLocal;
    const DevMember &m = member_of(a.ms, slot);
    const DevParams &Pm = a.ms.params[m.pIdx];
    const TileBox tb = tile_box(a.g, tile);
    const int tx = tile % a.g.ntx, ty = tile / a.g.ntx;
    const int bw = (tx == a.g.ntx - 1) ? m.rw - tb.x0 : a.g.blockW;
    const int bh = (ty == a.g.nty - 1) ? m.rh - tb.y0 : a.g.blockH;
    const int pair0 = blockIdx.y * a.pairsPerCta;
    // the CTA's row pairs; none when its results all lie outside the
    // member's region of interest (no transform, no extrema)
    int P = 2 * pair0 < bh ? min(a.pairsPerCta, (bh - 2 * pair0 + 1) >> 1) : 0;
    if (MODE == ROI && P > 0) {
        const int ya = tb.y0 + 2 * pair0, yb = tb.y0 + min(2 * (pair0 + P), bh);
        if (ya >= m.roiY1 || yb <= m.roiY0 || tb.x0 >= m.roiX1 || tb.x0 + bw <= m.roiX0) P = 0;
    }
    const int tid = threadIdx.x;
    unsigned int *bnd = a.bounds ? a.bounds + 2 * m.pIdx : nullptr;
    Ext e;
    ext_init(e);
    if (P > 0 && Pm.flat) {
        // a flat template scores 1 everywhere (impl.go:1137-1144)
        for (int rr = 0; rr < 2 * P && 2 * pair0 + rr < bh; rr++) {
            const int yy = tb.y0 + 2 * pair0 + rr;
            if (yy < m.roiY0 || yy >= m.roiY1) continue;
            for (int x = tid; x < bw; x += S::CTA) {
                const long long i = (long long)yy * m.rw + tb.x0 + x;
                if (a.ms.map) a.ms.map[i] = 1.f;
                if (tb.x0 + x >= m.roiX0 && tb.x0 + x < m.roiX1) ext_add(e, 1.f, i);
            }
        }
    } else if (P > 0) {
        e = line_pairs<L, FAST, MODE>(a, smem, m, Pm, tb, bw, bh, pair0, P, bnd);
    }
    // a CTA none of whose results passed its member's cuts has nothing to reduce
    if (__syncthreads_or(e.minI != LLONG_MAX || e.maxI != LLONG_MAX)) ext_block_reduce(e, shExt);
    if (MODE == TALLY && tid == 0 && P > 0 && !Pm.flat) {
        const unsigned int formed = *tally_word<L>();
        if (formed)
            atomicAdd(a.ms.formed + kTallyFormed + 16 * ((blockIdx.x + blockIdx.y) & (kTallySpread - 1)), formed);
    }
    if (tid == 0) {
        Partial &o = a.partials[m.partBase + a.partOffset + tileLocal * gridDim.y + blockIdx.y];
        o.minV = e.minV;
        o.maxV = e.maxV;
        o.minI = e.minI;
        o.maxI = e.maxI;
        if (bnd) {
            if (e.maxI != LLONG_MAX) atomicMax(bnd, ordered_key(e.maxV));
            if (e.minI != LLONG_MAX) atomicMax(bnd + 1, ordered_key(-e.minV));
        }
        __threadfence();
        isLast = atomicAdd(&a.counters[m.pIdx], 1) == a.nparts - 1;
    }
    __syncthreads();
    if (!isLast) return;
    __threadfence();
    ext_init(e);
    for (int i = tid; i < a.nparts; i += S::CTA) {
        const volatile Partial *p = a.partials + m.partBase + i;
        Ext o;
        o.minV = p->minV;
        o.maxV = p->maxV;
        o.minI = p->minI;
        o.maxI = p->maxI;
        ext_merge(e, o);
    }
    __syncthreads();
    ext_block_reduce(e, shExt);
    if (tid == 0) ext_store_result(e, m.rw, a.out + m.outIdx);
}

template <int L, bool FAST, Keep MODE>
void lines_one(const InvArgs &a, dim3 grid, cudaStream_t st) {
    const size_t smem = Lines<L>::SMEM + (MODE == TABLE || MODE == TALLY ? (kBlocksMax + 1) * sizeof(float) : 0);
    set_smem(k_inv_lines<L, FAST, MODE>, smem);
    launch_k(k_inv_lines<L, FAST, MODE>, grid, dim3(Lines<L>::CTA), smem, st, a);
}

template <int L>
void lines_form(const InvArgs &a, dim3 grid, cudaStream_t st) {
    const Keep k = a.ms.map ? ALL : (a.ms.anyRoi ? ROI : (a.ms.table ? LANES : SOLO));
    if (!a.ms.form)
        k == ALL ? lines_one<L, false, ALL>(a, grid, st)
        : k == ROI ? lines_one<L, false, ROI>(a, grid, st)
        : k == SOLO ? lines_one<L, false, SOLO>(a, grid, st) : lines_one<L, false, LANES>(a, grid, st);
    else if (a.ms.sat)
        a.ms.formed ? lines_one<L, true, TALLY>(a, grid, st) : lines_one<L, true, TABLE>(a, grid, st);
    else
        k == ALL ? lines_one<L, true, ALL>(a, grid, st)
        : k == ROI ? lines_one<L, true, ROI>(a, grid, st)
        : k == SOLO ? lines_one<L, true, SOLO>(a, grid, st) : lines_one<L, true, LANES>(a, grid, st);
}

}  // namespace

bool inv_lines_length(int log2n) { return log2n >= 7 && log2n <= 11; }

// Lines of a CTA at a time.
int inv_lines_cta(int log2n) { return log2n >= 10 ? 1 : 1 << (10 - log2n); }

void launch_inv_lines(const InvArgs &a, dim3 grid, cudaStream_t st) {
    switch (a.fc.log2n) {
        case 7: lines_form<7>(a, grid, st); break;
        case 8: lines_form<8>(a, grid, st); break;
        case 9: lines_form<9>(a, grid, st); break;
        case 10: lines_form<10>(a, grid, st); break;
        default: lines_form<11>(a, grid, st); break;
    }
}

}  // namespace cvm
