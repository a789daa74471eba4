// Neighbor-table kernels: full-grid init, fused top-k + compaction + table build, remap, check.
//
// Semantics follow the torch code of the reference backbone
// (opentad/models/backbones/vit_sparse_adapter_poguise.py: :1623-1670 init, :785-787 selection,
// :913-977 gather + remap); the algorithms do not: selection is an exact k-th-key search on
// order-preserving integer keys, compaction is a ballot/popc prefix scan, and the table is
// emitted straight from the kept set without materialising the old-to-new map in HBM.
#include <atomic>
#include <type_traits>

#include "common.cuh"

namespace svtad {

// float -> uint32 key with the same order as "a > b" on floats; every NaN maps to the largest
// key (torch.topk ranks NaN above all numbers); -0.0 and +0.0 map to the same key.
__device__ __forceinline__ uint32_t score_key(float f) {
    // the sum makes -0.0 +0.0 and any NaN the one that arithmetic returns, 0x7fffffff; it goes through another pipe than
    // compares and selects, which the builders' loops are short of
    const int b = __float_as_int(__fadd_rn(f, 0.0f));
    return (uint32_t)(b ^ (b >> 31 | (int)0x80000000));
}

// a score with that key (the canonical one of those that share it)
__device__ __forceinline__ float key_score(uint32_t key) {
    return __uint_as_float((key & 0x80000000u) ? key & 0x7FFFFFFFu : ~key);
}

// ------------------------------------------------------------------------------------------
// init
// ------------------------------------------------------------------------------------------
// Four entries per thread from 32-bit indices (UINT: fewer than 2^32 entries), one division for the row and one for its place
// in the grid.
template <typename UINT>
__global__ void table_init_kernel(int32_t* __restrict__ table, long total, int hw, int h, int w,
                                  int ksize, int kk) {
    pdl_wait();
    pdl_trigger();
    const UINT f0 = ((UINT)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (f0 >= (UINT)total) return;
    const int r = ksize >> 1;
    UINT row = f0 / (UINT)kk;
    int tap = (int)(f0 - row * (UINT)kk), p = (int)(row % (UINT)hw), y = p / w, x = p - y * w;
    int ty = tap / ksize, tx = tap - ty * ksize;
    int32_t v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int dy = ty - r, dx = tx - r;
        v[e] = ((unsigned)(y + dy) < (unsigned)h && (unsigned)(x + dx) < (unsigned)w) ? (int32_t)row + dy * w + dx : -1;
        if (++tx == ksize) {
            tx = 0;
            if (++ty == ksize) {
                ty = 0;
                ++row;
                if (++x == w) {
                    x = 0;
                    if (++y == h) y = 0;
                }
            }
        }
    }
    if (f0 + 3 < (UINT)total && (reinterpret_cast<uintptr_t>(table) & 15) == 0) {
        *reinterpret_cast<int4*>(table + f0) = make_int4(v[0], v[1], v[2], v[3]);
    } else {
        for (int e = 0; e < 4 && f0 + e < (UINT)total; ++e) table[f0 + e] = v[e];
    }
}

// ------------------------------------------------------------------------------------------
// build: one warp per segment (seg_len <= 32 * ITEMS)
// ------------------------------------------------------------------------------------------
// What bounds it: a warp's chain of dependent steps, one wave of them; 3 072 slices of 196 tokens, keep 25 %, in cycles: scores
// 2 900, threshold 3 100 by interpolation alone and about 1 000 behind the bins, rows 2 900 and about 2 000 with all of them staged
// at once.  Back to back 10.3 -> 7.8 us a call, of which 1.3 are the launch's early start; 160 slices 8.2 -> 5.5.
template <int KS>
__device__ __forceinline__ void tap_to_dydx(int tap, int ksize, int& dy, int& dx) {
    if constexpr (KS > 0) {
        dy = tap / KS - KS / 2;
        dx = tap % KS - KS / 2;
    } else {
        dy = tap / ksize - ksize / 2;
        dx = tap % ksize - ksize / 2;
    }
}

// floor(e / d) for e < 65536 with the host-computed multiplier ceil(2^32 / d)
__device__ __forceinline__ int div_magic(int e, uint32_t magic) { return (int)__umulhi((uint32_t)e, magic); }

template <int ITEMS, int KS>
__global__ void __launch_bounds__(256)
table_build_warp_kernel(const float* __restrict__ scores, int n_seg, int L, int k, int h, int w,
                        int ksize, uint32_t magic_w, uint32_t magic_hw, int32_t* __restrict__ kept_idx,
                        int32_t* __restrict__ table, int64_t* __restrict__ idx64) {
    constexpr int WARPS = 8;
    constexpr int CAP = ITEMS * 32;
    constexpr int KKMAX = (KS > 0) ? KS * KS : 49;
    __shared__ int32_t s_row[WARPS][CAP];            // a token's row in the table, -1 for those that go
    __shared__ int16_t s_pos[WARPS][CAP];
    constexpr int RR = KS == 3 ? 64 : KS == 5 ? 32 : 8;    // kept tokens whose rows are staged per round
    constexpr int STAGE = RR * KKMAX + 4 < 256 ? 256 : (RR * KKMAX + 7) & ~3;
    __shared__ __align__(16) int32_t s_out[WARPS][STAGE];  // staged table rows, written out with coalesced stores; before that, bins
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int seg = blockIdx.x * WARPS + wid;
    pdl_wait();            // no trigger: a successor's CTAs, resident beside these, would cost them more than it gains
    if (seg >= n_seg) return;
    const unsigned lt = (1u << lane) - 1u;
    const float* sc = scores + (long)seg * L;
    float score[ITEMS];
    uint32_t key[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) score[j] = __ldg(sc + min(j * 32 + lane, L - 1));
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) key[j] = j * 32 + lane < L ? score_key(score[j]) : 0u;   // 0 is below every real key
    // Threshold search between lo (at least k keys are >= lo) and hi (fewer are >= hi).  Of four candidates two come by
    // interpolation between the counts on the scores' own scale, one halves the interval on that scale and one on the
    // keys', which bounds the search for any input: 8 rounds for N(0,1) scores, 11 for softmax-like ones, where bit by
    // bit took 19, and none or one behind the bins.  Once a candidate splits off exactly k keys the kept set {key >= lo} is decided; if none does
    // (ties at the boundary) lo ends as the k-th largest key.
    uint32_t T = 0;
    bool decided = L == k;
    if (L != k) {
        uint32_t lo = 0, hi = 0xFFFFFFFFu, mx = 0;
        int n_lo = L, n_hi = 0;
        {
            uint32_t mn = 0xFFFFFFFFu;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                mx = max(mx, key[j]);
                if (j * 32 + lane < L) mn = min(mn, key[j]);
            }
            lo = __reduce_min_sync(0xffffffffu, mn);
            mx = __reduce_max_sync(0xffffffffu, mx);
        }
        if (mx == 0xFFFFFFFFu) {          // NaNs: they are kept first
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) n_hi += key[j] == mx;
            n_hi = __reduce_add_sync(0xffffffffu, n_hi);
            if (n_hi >= k) lo = mx;
        } else {
            hi = mx + 1;
        }
        // Where the scores are finite and not all alike, 256 bins of equal width between the least and the largest say which
        // few keys the threshold is among: 1 or 2 of 196 normal scores.
        const float f_mn = key_score(lo), range = key_score(mx) - f_mn;
        if (hi == mx + 1 && range > 1e-30f && range < 1e30f && f_mn > -1e30f) {
            int32_t* bins = s_out[wid];
            *reinterpret_cast<int4*>(bins + 8 * lane) = make_int4(0, 0, 0, 0);
            *reinterpret_cast<int4*>(bins + 8 * lane + 4) = make_int4(0, 0, 0, 0);
            __syncwarp();
            // the bin as the low bits of a sum (rounded to nearest; every operation is monotone)
            const float scale = __fdividef(255.0f, range);
            auto bin_of = [&](float f) { return __float_as_int(__fmaf_rn(f - f_mn, scale, 8388608.0f)) & 0x1FF; };
            int bin[ITEMS];
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                bin[j] = j * 32 + lane < L ? min(bin_of(score[j]), 255) : -1;
                if (bin[j] >= 0) atomicAdd(bins + bin[j], 1);
            }
            __syncwarp();
            const int top = 8 * (31 - lane);           // a lane's eight bins, the highest first
            const int4 b_lo = *reinterpret_cast<const int4*>(bins + top), b_hi = *reinterpret_cast<const int4*>(bins + top + 4);
            const int v[8] = {b_hi.w, b_hi.z, b_hi.y, b_hi.x, b_lo.w, b_lo.z, b_lo.y, b_lo.x};
            int mine = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) mine += v[q];
            int above = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, above, d);
                if (lane >= d) above += t;
            }
            const int owner = __ffs(__ballot_sync(0xffffffffu, above >= k)) - 1;
            above -= mine;
            int at = top + 7, count = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (count == 0 && above + v[q] >= k) count = v[q];
                if (count == 0) { above += v[q]; --at; }
            }
            at = __shfl_sync(0xffffffffu, at, owner);
            n_hi = __shfl_sync(0xffffffffu, above, owner);
            n_lo = n_hi + __shfl_sync(0xffffffffu, count, owner);
            uint32_t in = 0xFFFFFFFFu, over = hi;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                if (bin[j] == at) in = min(in, key[j]);
                if (bin[j] > at) over = min(over, key[j]);
            }
            lo = __reduce_min_sync(0xffffffffu, in);
            hi = __reduce_min_sync(0xffffffffu, over);
            decided = n_lo == k;
            __syncwarp();
        }
        for (int round = 0; !decided && hi - lo > 1; ++round) {
            uint32_t cand = lo + (hi - lo) / 2;
            if ((round & 3) != 3) {
                const float f_lo = key_score(lo), f_hi = key_score(hi);
                const float at = (round & 3) == 2 ? 0.5f : __fdividef((float)(n_lo - k) + 0.5f, (float)(n_lo - n_hi));
                const uint32_t by_value = score_key(f_lo + (f_hi - f_lo) * at);
                if (by_value > lo && by_value < hi) cand = by_value;       // not for an infinite or NaN value
            }
            int c = 0;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) c += (key[j] >= cand);
            c = __reduce_add_sync(0xffffffffu, c);
            if (c >= k) { lo = cand; n_lo = c; } else { hi = cand; n_hi = c; }
            decided = c == k;
        }
        T = lo;
    }

    const int base = seg * k;                          // row numbers fit 31 bits
    int run_keep = 0;
    if (decided) {
        unsigned km[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) km[j] = __ballot_sync(0xffffffffu, j * 32 + lane < L && key[j] >= T);
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const int e = j * 32 + lane, rank = run_keep + __popc(km[j] & lt);
            const bool keep = (km[j] >> lane) & 1u;
            if (e < L) s_row[wid][e] = keep ? base + rank : -1;
            if (keep) s_pos[wid][rank] = (int16_t)e;
            run_keep += __popc(km[j]);
        }
    } else {
        int gt = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) gt += (key[j] > T);
        const int need_ties = k - __reduce_add_sync(0xffffffffu, gt);   // >= 1 ties at the threshold are kept, lowest index first
        int run_tie = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const int e = j * 32 + lane;
            const bool valid = e < L, eq = valid && key[j] == T;
            const unsigned eqm = __ballot_sync(0xffffffffu, eq);
            const bool keep = (valid && key[j] > T) || (eq && run_tie + __popc(eqm & lt) < need_ties);
            const unsigned km = __ballot_sync(0xffffffffu, keep);
            const int rank = run_keep + __popc(km & lt);
            if (valid) s_row[wid][e] = keep ? base + rank : -1;
            if (keep) s_pos[wid][rank] = (int16_t)e;
            run_tie += __popc(eqm);
            run_keep += __popc(km);
        }
    }
    __syncwarp();
    const int hw = h * w;

    if (kept_idx != nullptr)
        for (int r = lane; r < k; r += 32) kept_idx[base + r] = s_pos[wid][r];
    if (idx64 != nullptr)
        for (int r = lane; r < k; r += 32) idx64[base + r] = s_pos[wid][r];
    if (table == nullptr) return;

    // A lane per kept token (two in turn for 3 x 3) computes its K*K entries into shared memory, placed so that the rows, which
    // are contiguous in the table, leave with 16-byte loads and stores.
    const int KK = (KS > 0) ? KS * KS : ksize * ksize;
    const int RN = KS > 0 ? RR : min(RR, RR * KKMAX / KK);      // stencils beyond 7 x 7: as many rows as fit (15 x 15: one)
    const bool vectors = (reinterpret_cast<uintptr_t>(table) & 15) == 0;
    int32_t* so = s_out[wid];
    for (int r0 = 0; r0 < k; r0 += RN) {
        const long g0 = ((long)base + r0) * KK;            // first table element of this round
        const int shift = (int)(g0 & 3);
#pragma unroll
        for (int q = 0; q < (RR + 31) / 32; ++q) {
            const int rl = q * 32 + lane, r = r0 + rl;
            if (rl < RN && r < k) {
                const int p = s_pos[wid][r], g = hw == 1 ? 0 : p - div_magic(p, magic_hw) * hw;
                const int y = w == 1 ? g : div_magic(g, magic_w), x = g - y * w;
                int32_t* mine = so + shift + rl * KK;
                auto entry = [&](int tap, int dy, int dx) {
                    int32_t v = -1;
                    if ((unsigned)(y + dy) < (unsigned)h && (unsigned)(x + dx) < (unsigned)w) v = s_row[wid][p + dy * w + dx];
                    mine[tap] = v;
                };
                if constexpr (KS > 0) {
#pragma unroll
                    for (int tap = 0; tap < KS * KS; ++tap) entry(tap, tap / KS - KS / 2, tap % KS - KS / 2);
                } else {
                    for (int tap = 0; tap < KK; ++tap) entry(tap, tap / ksize - ksize / 2, tap % ksize - ksize / 2);
                }
            }
        }
        __syncwarp();
        const int end = shift + ((k - r0) < RN ? (k - r0) : RN) * KK;
        int32_t* out = table + (g0 - shift);
        for (int o = 4 * lane; o < end; o += 128) {
            if (vectors && o >= shift && o + 4 <= end) {
                *reinterpret_cast<int4*>(out + o) = *reinterpret_cast<const int4*>(so + o);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (o + e >= shift && o + e < end) out[o + e] = so[o + e];
            }
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------------------------------
// build: several CTAs per segment (seg_len > 256: a clip, or a long batch row)
// ------------------------------------------------------------------------------------------
// What bounds it: latency, and the issue slots of the few SMs that write the rows out.  A clip of 15 680 scores is 60 KB
// and its table 340 KB, but every step of the selection (radix passes, prefix sums) waits for the one before.  So the CTAs
// of a segment share nothing: each makes the whole selection from all scores, in its registers and its own shared memory,
// and writes the rows of its part of the tokens; there are as many CTAs as half the GPU holds, and the next round's take
// the other half.  Measured in cycles of a CTA, 15 680 -> 9 408 tokens, two clips: scores 2 900, radix passes 5 700, ranks 1 600,
// rows 3 400.  Clusters of up to eight CTAs that shared the selection through distributed shared memory, one barrier per
// radix pass, took 2 900, 10 900, 3 700 and 7 800; three rounds of two 160-frame clips 42 us where these kernels take 24.
//   * scores are read once and stay in registers as order-preserving keys; radix passes of 12, 10 and 10 bits, the last two
//     over the keys of the first one's bin, and only until every key of a bin is kept;
//   * what is kept is one bit per token: after a scan over the words rank(token) is a word, a mask and a popcount;
//   * the rows of a word's kept tokens are contiguous in the output: warps write them with coalesced stores, several per
//     word where a CTA has few.
// Segments beyond 16 384 tokens keep the clusters: their keys do not fit one CTA's registers.
constexpr int SEG_THREADS = 1024, SEG_WARPS = SEG_THREADS / 32, SEG_MAX = 51200, SEG_ALONE = 16384;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t in_cta(uint32_t saddr, int cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(cta));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ int warp_incl_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += t;
    }
    return v;
}
// exclusive prefix sum of v over the block in thread order (all threads call)
__device__ __forceinline__ int block_excl_scan(int v, int* s_w) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int incl = warp_incl_scan(v);
    __syncthreads();               // s_w free for reuse
    if (lane == 31) s_w[wid] = incl;
    __syncthreads();
    return __reduce_add_sync(0xffffffffu, lane < wid ? s_w[lane] : 0) + incl - v;
}

struct SegArgs {
    const float* scores;
    int L, k, h, w, ksize;
    uint32_t magic_w, magic_hw, magic_ks;
    int kk;
    int32_t* kept_idx;
    int32_t* table;
    int64_t* idx64;
    const int32_t* table_in;               // rows to renumber (a later pruning round); null: the grid's own
    int staged;                            // this CTA's rows of table_in fit its shared memory
    int words;                             // of 32 tokens per CTA
    int ctas;                              // per segment
};

// The rows of a later round start their trip to shared memory; source and target stay equally aligned.
__device__ __forceinline__ int seg_shift(const int32_t* rows_in) { return (int)((reinterpret_cast<uintptr_t>(rows_in) >> 2) & 3); }
__device__ __forceinline__ void seg_stage_rows(const int32_t* rows_in, int n_rows, int kk, int32_t* s_rows) {
    const int shift = seg_shift(rows_in), total = n_rows * kk, lead = min(total, (4 - shift) & 3), vec = (total - lead) >> 2, tid = threadIdx.x;
    auto copy = [&](int f, int bytes) {
        const uint32_t dst = smem_addr(s_rows + shift + f);
        if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(rows_in + f) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(rows_in + f) : "memory");
    };
    if (tid < lead) copy(tid, 4);
    for (int v = tid; v < vec; v += SEG_THREADS) copy(lead + 4 * v, 16);
    for (int f = lead + 4 * vec + tid; f < total; f += SEG_THREADS) copy(f, 4);
}

// s_rank: per word its kept bits and the output row of its first kept token.  A warp writes part `part` of `parts` of a word's
// kept positions and table rows; `in`: the word's rows of the previous table.
__device__ __forceinline__ void seg_write_word(const SegArgs& p, const uint2* s_rank, uint32_t* list, int seg, int word, int part,
                                               int parts, const int32_t* in) {
    const int lane = threadIdx.x & 31, hw = p.h * p.w, r0 = p.ksize >> 1, seg0 = seg * p.L;      // row numbers fit 31 bits
    const uint2 rk = s_rank[word];
    const int e = word * 32 + lane;
    auto renumbered = [&](unsigned loc) -> int32_t {
        const uint2 r = s_rank[loc >> 5];
        const uint32_t below = r.x << (31 - (loc & 31));        // the token's own bit on top
        return below >> 31 ? (int32_t)(r.y + __popc(below) - 1) : -1;
    };
    if ((rk.x >> lane) & 1u) {
        const int r = __popc(rk.x & ((1u << lane) - 1u));
        if (part == 0 && p.kept_idx != nullptr) p.kept_idx[rk.y + r] = e;
        if (part == 0 && p.idx64 != nullptr) p.idx64[rk.y + r] = e;
        const int q = hw == 1 ? 0 : e - div_magic(e, p.magic_hw) * hw;
        const int y = p.w == 1 ? q : div_magic(q, p.magic_w), x = q - y * p.w;
        list[r] = (uint32_t)lane | (uint32_t)(y & 0xFF) << 8 | (uint32_t)(x & 0xFF) << 16;
    }
    if (p.table == nullptr) return;
    __syncwarp();
    const int kk = p.kk, entries = __popc(rk.x) * kk, step = 32 * parts, d_row = step / kk, d_tap = step - d_row * kk;
    int32_t* out = p.table + (long)rk.y * kk;
    int r = (part * 32 + lane) / kk, tap = part * 32 + lane - r * kk;
    auto advance = [&] {
        r += d_row;
        tap += d_tap;
        if (tap >= kk) { tap -= kk; ++r; }
    };
    if (p.table_in != nullptr) {
        // later round: the kept rows of the previous table, renumbered
#pragma unroll 4
        for (int f = part * 32 + lane; f < entries; f += step) {
            const int32_t old = in[(int)(list[r] & 31u) * kk + tap];
            const unsigned loc = (unsigned)(old - seg0);
            out[f] = old >= 0 && loc < (unsigned)p.L ? renumbered(loc) : -1;
            advance();
        }
    } else {
        for (int f = part * 32 + lane; f < entries; f += step) {
            const int ty = p.ksize == 1 ? tap : div_magic(tap, p.magic_ks);
            const int dy = ty - r0, dx = tap - ty * p.ksize - r0;
            const uint32_t it = list[r];
            const int y = (int)(it >> 8 & 0xFFu) + dy, x = (int)(it >> 16) + dx;
            out[f] = (unsigned)y < (unsigned)p.h && (unsigned)x < (unsigned)p.w ? renumbered(word * 32 + (int)(it & 31u) + dy * p.w + dx) : -1;
            advance();
        }
    }
    __syncwarp();
}

constexpr int SEG_FEW = 2048;              // keys of a bin that are gathered

// ITEMS = words per warp: all of the segment's, word 32 j + warp for j < ITEMS
template <int ITEMS>
__global__ void __launch_bounds__(SEG_THREADS)
table_select_kernel(const SegArgs p) {
    extern __shared__ __align__(16) int32_t s_rows[];     // this CTA's rows of table_in, if they fit
    constexpr int WORDS = ITEMS * SEG_WARPS;
    __shared__ __align__(16) int s_hist[4096 + 2 * 1024];
    __shared__ int s_found[3], s_w[SEG_WARPS];
    __shared__ uint32_t s_from[WORDS], s_eq[WORDS];        // keys from the threshold on, and equal to it
    __shared__ uint2 s_rank[WORDS];                        // see seg_write_word
    __shared__ uint32_t s_few[SEG_FEW];
    __shared__ int s_n;
    __shared__ uint32_t s_list[SEG_WARPS][32];             // per warp: its word's kept tokens, lane | y << 8 | x << 16
    const int seg = blockIdx.x / p.ctas, cta = blockIdx.x - seg * p.ctas;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, L = p.L;
    const int n_words = (L + 31) >> 5, w_begin = cta * p.words, w_end = min(n_words, w_begin + p.words);
#pragma unroll
    for (int q = 0; q < 6; ++q) s_hist[q * 1024 + tid] = 0;
    if (tid == 0) s_n = 0;
    pdl_wait();
    pdl_trigger();
    const float* sc = p.scores + (long)seg * L;
    float score[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int e = (j * SEG_WARPS + wid) * 32 + lane;
        score[j] = __ldg(sc + (e < L ? e : 0));
    }
    const int32_t* rows_in = p.table_in != nullptr ? p.table_in + ((long)seg * L + w_begin * 32) * p.kk : nullptr;
    if (p.staged) seg_stage_rows(rows_in, max(0, min(L, w_end * 32) - w_begin * 32), p.kk, s_rows);
    uint32_t key[ITEMS];       // 0 behind the segment's end: below every real key (those begin at 0x007fffff)
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) key[j] = (j * SEG_WARPS + wid) * 32 + lane < L ? score_key(score[j]) : 0u;
    __syncthreads();

    // (1) radix select of the k-th largest key: the bin that holds the need-th of the keys that match so far, from the top
    uint32_t T = 0;
    int need = p.k, at_T = 0;
    auto find = [&](const int* hist, auto quads) {         // 1024 * quads bins, by eight warps (all threads call)
        __syncthreads();
        if (tid < 256) {
            constexpr int Q = decltype(quads)::value;
            int4 c[Q];
            int sum = 0;
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                c[q] = reinterpret_cast<const int4*>(hist)[(255 - tid) * Q + q];
                sum += c[q].x + c[q].y + c[q].z + c[q].w;
            }
            int above = warp_incl_scan(sum);
            if (lane == 31) s_w[wid] = above;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            above += __reduce_add_sync(0xffffffffu, lane < wid ? s_w[lane] : 0) - sum;      // keys in higher bins
            if (above < need && above + sum >= need) {
                int bin = ((255 - tid) * Q + Q) * 4 - 1, count = 0;
#pragma unroll
                for (int q = Q - 1; q >= 0; --q) {
                    const int v[4] = {c[q].w, c[q].z, c[q].y, c[q].x};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (count == 0 && above + v[e] >= need) count = v[e];
                        if (count == 0) { above += v[e]; --bin; }
                    }
                }
                s_found[0] = bin;
                s_found[1] = need - above;
                s_found[2] = count;
            }
        }
        __syncthreads();
        need = s_found[1];
        at_T = s_found[2];
        return (uint32_t)s_found[0];
    };
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) atomicAdd(&s_hist[key[j] >> 20], 1);
    T = find(s_hist, std::integral_constant<int, 4>());
    // The bin's keys, a few hundred of 15 680 normal ones, are gathered for the two passes that are left; there is nothing to
    // be found out once every key of a bin is kept.
    int shift = 20;
    if (at_T != need) {
        const bool few = at_T <= SEG_FEW;
        if (few) {
            int mine = 0;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) mine += key[j] >> 20 == T;
            const int incl = warp_incl_scan(mine);
            int at = 0;
            if (lane == 31) at = atomicAdd(&s_n, incl);
            at = __shfl_sync(0xffffffffu, at, 31) + incl - mine;
            if (mine > 0) {
#pragma unroll
                for (int j = 0; j < ITEMS; ++j)
                    if (key[j] >> 20 == T) s_few[at++] = key[j];
            }
            __syncthreads();
        }
        const int n_few = few ? at_T : 0;
#pragma unroll 1
        for (int pass = 0; pass < 2 && at_T != need; ++pass) {
            int* hist = s_hist + 4096 + 1024 * pass;
            shift -= 10;
            auto count = [&](uint32_t key) {
                if (key >> shift >> 10 == T) atomicAdd(&hist[key >> shift & 1023], 1);
            };
            if (few) {
                for (int e = tid; e < n_few; e += SEG_THREADS) count(s_few[e]);
            } else {
#pragma unroll
                for (int j = 0; j < ITEMS; ++j) count(key[j]);
            }
            T = T << 10 | find(hist, std::integral_constant<int, 1>());
        }
    }
    T <<= shift;

    // (2) kept bits: keys from T on; where not every key equal to T is kept, lower tokens first
    const bool ties = at_T != need;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t from = __ballot_sync(0xffffffffu, key[j] >= T);
        if (lane == 0) s_from[j * SEG_WARPS + wid] = from;
    }
    if (ties) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t eq = __ballot_sync(0xffffffffu, key[j] == T);
            if (lane == 0) s_eq[j * SEG_WARPS + wid] = eq;
        }
    }
    __syncthreads();
    {
        uint32_t kept = tid < n_words ? s_from[tid] : 0u;
        if (ties) {
            uint32_t eq = tid < n_words ? s_eq[tid] : 0u;
            kept &= ~eq;
            const int room = max(0, need - block_excl_scan(__popc(eq), s_w));
            while (__popc(eq) > room) eq &= ~(0x80000000u >> __clz(eq));         // drop the highest
            kept |= eq;
        }
        const int before = block_excl_scan(__popc(kept), s_w);
        if (tid < n_words) s_rank[tid] = make_uint2(kept, seg * p.k + before);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // (3) kept positions and table rows of this CTA's words, each by as many warps as there are to spare
    const int parts = max(1, SEG_WARPS / p.words);
    for (int u = wid; u < (w_end - w_begin) * parts; u += SEG_WARPS) {
        const int at = u / parts, word = w_begin + at;
        const int32_t* in = p.staged ? s_rows + seg_shift(rows_in) + at * 32 * p.kk : rows_in + at * 32 * (long)p.kk;
        seg_write_word(p, s_rank, s_list[wid], seg, word, u - at * parts, parts, in);
    }
}

// Segments beyond SEG_ALONE: eight CTAs of a cluster hold seven words per warp of it and add their histograms up through
// distributed shared memory, each for itself; every CTA gets the whole bit set.
constexpr int SEG_G = 8, SEG_ITEMS = 7, SEG_WORDS = SEG_MAX / 32;

__global__ void __launch_bounds__(SEG_THREADS)
table_select_cluster_kernel(const SegArgs p) {
    extern __shared__ __align__(16) int32_t s_rows[];     // this CTA's rows of table_in, if they fit
    __shared__ int s_hist[4][256];
    __shared__ int s_found[3];
    __shared__ uint32_t s_keep[SEG_WORDS], s_eq[SEG_WORDS];
    __shared__ uint2 s_rank[SEG_WORDS];
    __shared__ uint32_t s_list[SEG_WARPS][32];
    __shared__ int s_w[SEG_WARPS];
    const int seg = blockIdx.x / SEG_G, cta = blockIdx.x % SEG_G, L = p.L;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int n_words = (L + 31) >> 5, w_begin = cta * p.words, w_end = min(n_words, w_begin + p.words);
    const float* sc = p.scores + (long)seg * L;
    pdl_wait();
    pdl_trigger();

    uint32_t key[SEG_ITEMS];
#pragma unroll
    for (int j = 0; j < SEG_ITEMS; ++j) {
        const int word = w_begin + wid + 32 * j, e = word * 32 + lane;
        key[j] = word < w_end && e < L ? score_key(__ldg(sc + e)) : 0u;     // 0 is below every real key
    }
    s_hist[tid >> 8][tid & 255] = 0;
    const int32_t* rows_in = p.table_in != nullptr ? p.table_in + ((long)seg * L + w_begin * 32) * p.kk : nullptr;
    if (p.staged) seg_stage_rows(rows_in, max(0, min(L, w_end * 32) - w_begin * 32), p.kk, s_rows);
    __syncthreads();

    // (1) radix select of the k-th largest key, one byte per pass, most significant first
    uint32_t T = 0, mask = 0;
    int need = p.k, at_T = 0;
#pragma unroll 1
    for (int pass = 3; pass >= 0; --pass) {
#pragma unroll
        for (int j = 0; j < SEG_ITEMS; ++j) {
            const int word = w_begin + wid + 32 * j;
            const bool in = word < w_end && word * 32 + lane < L && (key[j] & mask) == T;
            const int bin = (key[j] >> (8 * pass)) & 255;
            if (pass == 3) {
                // sign and exponent fall into a handful of bins: one add per bin and warp
                const unsigned same = __match_any_sync(0xffffffffu, in ? bin : 256);
                if (in && (same & lt) == 0) atomicAdd(&s_hist[3][bin], __popc(same));
            } else if (in) {
                atomicAdd(&s_hist[pass][bin], 1);
            }
        }
        cluster_sync();
        // thread t adds up bin 255 - t; an inclusive scan over the bins in descending order names the one that holds
        // the need-th key (always found: matching keys >= need)
        int c = 0, incl = 0;
        if (tid < 256) {
            const uint32_t mine = smem_addr(&s_hist[pass][255 - tid]);
#pragma unroll
            for (int g = 0; g < SEG_G; ++g) {
                int v;
                asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(in_cta(mine, g)) : "memory");
                c += v;
            }
            incl = warp_incl_scan(c);
            if (lane == 31) s_w[wid] = incl;
        }
        __syncthreads();
        if (tid < 256) {
            for (int q = 0; q < wid; ++q) incl += s_w[q];
            if (incl >= need && incl - c < need) {
                s_found[0] = 255 - tid;
                s_found[1] = need - (incl - c);
                s_found[2] = c;
            }
        }
        __syncthreads();
        T |= (uint32_t)s_found[0] << (8 * pass);
        need = s_found[1];
        at_T = s_found[2];
        mask |= 0xFFu << (8 * pass);
    }

    // (2) kept bits: keys above T, and of those equal to T the first `need`
#pragma unroll
    for (int j = 0; j < SEG_ITEMS; ++j) {
        const int word = w_begin + wid + 32 * j;
        const bool valid = word < w_end && word * 32 + lane < L;
        const uint32_t gt = __ballot_sync(0xffffffffu, valid && key[j] > T);
        const uint32_t eq = __ballot_sync(0xffffffffu, valid && key[j] == T);
        if (word < w_end && lane < SEG_G) {
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(in_cta(smem_addr(&s_keep[word]), lane)), "r"(gt) : "memory");
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(in_cta(smem_addr(&s_eq[word]), lane)), "r"(eq) : "memory");
        }
    }
    cluster_sync();                    // also the last access to another CTA's shared memory
    constexpr int WPT = (SEG_WORDS + SEG_THREADS - 1) / SEG_THREADS;     // words per thread in the scans
    {
        int ties = 0;
        if (at_T != need) {            // not every key equal to T is kept: lower tokens first
            int c = 0;
#pragma unroll
            for (int q = 0; q < WPT; ++q)
                if (tid * WPT + q < n_words) c += __popc(s_eq[tid * WPT + q]);
            ties = block_excl_scan(c, s_w);
        }
        uint32_t kw[WPT];
        int c = 0;
#pragma unroll
        for (int q = 0; q < WPT; ++q) {
            const int word = tid * WPT + q;
            kw[q] = 0;
            if (word < n_words) {
                uint32_t eq = s_eq[word];
                int room = at_T != need ? max(0, need - ties) : 32;
                ties += __popc(eq);
                while (__popc(eq) > room) eq &= ~(0x80000000u >> __clz(eq));     // drop the highest
                kw[q] = s_keep[word] | eq;
                c += __popc(kw[q]);
            }
        }
        int before = block_excl_scan(c, s_w);
#pragma unroll
        for (int q = 0; q < WPT; ++q) {
            const int word = tid * WPT + q;
            if (word < n_words) { s_rank[word] = make_uint2(kw[q], seg * p.k + before); before += __popc(kw[q]); }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // (3) a word's kept positions and table rows
    for (int word = w_begin + wid; word < w_end; word += SEG_WARPS) {
        const int at = word - w_begin;
        const int32_t* in = p.staged ? s_rows + seg_shift(rows_in) + at * 32 * p.kk : rows_in + at * 32 * (long)p.kk;
        seg_write_word(p, s_rank, s_list[wid], seg, word, 0, 1, in);
    }
}

// floor(e / d) = umulhi(e, magic) for e < 65536 (see div_magic)
static uint32_t magic_of(int d) { return (uint32_t)((0x100000000ull + d - 1) / d); }

static int segment_launch(const float* scores, int n_seg, int L, int k, int h, int w, int ksize, int kk, int32_t* kept_idx,
                          int32_t* table, int64_t* idx64, const int32_t* table_in, cudaStream_t s) {
    const int n_words = (L + 31) / 32;
    int words, ctas;
    if (L <= SEG_ALONE) {
        // Half the GPU's SMs for all segments together where that leaves a warp no more than one word (three rounds of eight
        // 80-frame clips: 27.7 us, on all SMs 30.2), else all of them (24 clips of 80 slices: 54 us, on half 73); at least
        // four words, of up to eight warps each, per CTA.
        const int half = tc_num_sms() / 2;
        const int want = ((long)n_words * n_seg <= (long)half * SEG_WARPS ? half : 2 * half) / n_seg;
        words = want > 1 ? (n_words + want - 1) / want : n_words;
        if (words < 4) words = 4;
        ctas = (n_words + words - 1) / words;
    } else {
        words = (n_words + SEG_G - 1) / SEG_G;
        ctas = SEG_G;
    }
    auto kern = L <= 2048 ? table_select_kernel<2> : L <= 4096 ? table_select_kernel<4> : L <= 8192 ? table_select_kernel<8>
                : L <= SEG_ALONE ? table_select_kernel<16> : table_select_cluster_kernel;
    // rows of the previous table wait in shared memory while they leave room for it
    const size_t rows = (size_t)words * 32 * kk * sizeof(int32_t) + 16;
    const int staged = table_in != nullptr && rows <= 176 * 1024;
    if (staged) {
        int rc = tc_ensure_smem(reinterpret_cast<const void*>(kern), 176 * 1024);
        if (rc) return rc;
    }
    const SegArgs p{scores, L, k, h, w, ksize, magic_of(w), magic_of(h * w), magic_of(ksize), kk, kept_idx, table, idx64, table_in, staged, words, ctas};
    SV_CUDA(launch_pdl(kern, dim3((unsigned)(n_seg * ctas)), dim3(SEG_THREADS), staged ? rows : 0, s, L <= SEG_ALONE ? 1 : SEG_G, p));
    return SVTAD_OK;
}

// ------------------------------------------------------------------------------------------
// remap
// ------------------------------------------------------------------------------------------
__global__ void remap_scatter_kernel(const int64_t* __restrict__ idx, int32_t* __restrict__ map,
                                     int B, int n_prev, int n_new) {
    long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (t >= (long)B * n_new) return;
    int b = (int)(t / n_new);
    int64_t p = idx[t];
    if (p < 0 || p >= n_prev) return;       // ignored, never written out of range
    map[(long)b * n_prev + p] = (int32_t)t;  // t == b*n_new + j
}

__global__ void remap_gather_kernel(const int32_t* __restrict__ table_in,
                                    const int64_t* __restrict__ idx,
                                    const int32_t* __restrict__ map, int32_t* __restrict__ out,
                                    int B, int n_prev, int n_new, int kk) {
    long f = blockIdx.x * (long)blockDim.x + threadIdx.x;
    long total = (long)B * n_new * kk;
    if (f >= total) return;
    long row = f / kk;
    int tap = (int)(f - row * kk);
    int b = (int)(row / n_new);
    int64_t p = idx[row];
    int32_t v = -1;
    if (p >= 0 && p < n_prev) {
        int32_t old = __ldg(table_in + ((long)b * n_prev + p) * kk + tap);
        if (old >= 0 && (long)old < (long)B * n_prev) v = map[old];
    }
    out[f] = v;
}

// ------------------------------------------------------------------------------------------
// check
// ------------------------------------------------------------------------------------------
__global__ void table_check_kernel(const int32_t* __restrict__ nbr, long n, int kk, int tpb,
                                   int32_t* __restrict__ status) {
    long f = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (f >= n * kk) return;
    long i = f / kk;
    int k = (int)(f - i * kk);
    int32_t j = __ldg(nbr + f);
    if (j == -1) return;
    long off = tpb > 0 ? (i / tpb) * (long)tpb : 0;
    long jj = (long)j + off;
    int bad = 0;
    if (j < -1 || jj < 0 || jj >= n) {
        bad = SVTAD_TABLE_OUT_OF_RANGE | SVTAD_TABLE_ASYMMETRIC;
    } else {
        int32_t back = __ldg(nbr + jj * kk + (kk - 1 - k));
        long off2 = tpb > 0 ? (jj / tpb) * (long)tpb : 0;
        if (back == -1 || (long)back + off2 != i) bad = SVTAD_TABLE_ASYMMETRIC;
    }
    if (bad && ((*reinterpret_cast<volatile int32_t*>(status)) & bad) != bad) atomicOr(status, bad);
}

}  // namespace svtad

using namespace svtad;

// ------------------------------------------------------------------------------------------
// C ABI
// ------------------------------------------------------------------------------------------
extern "C" int svtad_table_init(int B, int T, int h, int w, int ksize, int32_t* table,
                                void* stream) {
    SV_CHECK_ARG(B >= 0 && T >= 0 && h > 0 && w > 0, "svtad_table_init: bad grid %d x %d x %d x %d", B, T, h, w);
    SV_CHECK_ARG(ksize >= 1 && (ksize & 1), "svtad_table_init: ksize must be odd, got %d", ksize);
    long rows = (long)B * T * h * w;
    SV_CHECK_ARG(rows < (1l << 31), "svtad_table_init: %ld rows do not fit int32 indices", rows);
    if (rows == 0) return SVTAD_OK;
    SV_CHECK_ARG(table != nullptr, "svtad_table_init: table is null");
    long total = rows * ksize * ksize;
    long threads = (total + 3) / 4;
    auto kern = total < (1l << 32) - 4096 ? table_init_kernel<uint32_t> : table_init_kernel<uint64_t>;
    SV_CUDA(launch_pdl(kern, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, (cudaStream_t)stream, 1, table,
                       total, h * w, h, w, ksize, ksize * ksize));
    return SVTAD_OK;
}

static int table_build_impl(const float* scores, int n_seg, int seg_len, int k, int h, int w,
                            int ksize, int32_t* kept_idx, int32_t* table, int64_t* idx64,
                            void* stream, const char* who) {
    SV_CHECK_ARG(n_seg >= 0 && seg_len > 0, "%s: bad n_seg=%d seg_len=%d", who, n_seg, seg_len);
    SV_CHECK_ARG(k >= 0 && k <= seg_len, "%s: k_keep=%d outside [0, %d]", who, k, seg_len);
    if (table != nullptr) {
        SV_CHECK_ARG(h > 0 && w > 0 && seg_len % (h * w) == 0,
                     "%s: seg_len=%d is not a multiple of h*w=%d*%d", who, seg_len, h, w);
        SV_CHECK_ARG(ksize >= 1 && (ksize & 1) && ksize <= 15, "%s: ksize must be odd and <= 15, got %d", who, ksize);
        SV_CHECK_ARG(h < 256 && w < 256, "%s: grid side must be < 256", who);
    } else {
        h = seg_len; w = 1; ksize = 1;
    }
    SV_CHECK_ARG((long)n_seg * k < (1l << 31), "%s: n_seg*k_keep does not fit int32 indices", who);
    if (n_seg == 0 || k == 0) return SVTAD_OK;
    SV_CHECK_ARG(scores != nullptr, "%s: scores is null", who);
    cudaStream_t s = (cudaStream_t)stream;
    if (seg_len <= 256) {
        unsigned grid = (unsigned)((n_seg + 7) / 8);
        const uint32_t mw = (uint32_t)((0x100000000ull + w - 1) / w), mhw = (uint32_t)((0x100000000ull + h * w - 1) / (h * w));
        auto kern = ksize == 3 ? table_build_warp_kernel<8, 3> : ksize == 5 ? table_build_warp_kernel<8, 5> : table_build_warp_kernel<8, 0>;
        SV_CUDA(launch_pdl(kern, dim3(grid), dim3(256), 0, s, 1, scores, n_seg, seg_len, k, h, w, ksize, mw, mhw, kept_idx, table, idx64));
        return SVTAD_OK;
    }
    SV_CHECK_ARG(table == nullptr || kept_idx != nullptr, "%s: kept_idx is required with a table", who);
    if (seg_len > SEG_MAX)
        return set_error(SVTAD_ERR_UNSUPPORTED, "%s: seg_len=%d exceeds the %d-token segment limit", who, seg_len, SEG_MAX);
    return segment_launch(scores, n_seg, seg_len, k, h, w, ksize, ksize * ksize, kept_idx, table, idx64, nullptr, s);
}

extern "C" int svtad_table_build(const float* scores, int n_seg, int seg_len, int k_keep, int h,
                                 int w, int ksize, int32_t* kept_idx, int32_t* table,
                                 void* stream) {
    SV_CHECK_ARG(k_keep >= 0 && k_keep <= seg_len, "svtad_table_build: k_keep=%d outside [0, %d]", k_keep, seg_len);
    SV_CHECK_ARG(n_seg <= 0 || k_keep == 0 || (kept_idx != nullptr && table != nullptr),
                 "svtad_table_build: kept_idx / table is null");
    return table_build_impl(scores, n_seg, seg_len, k_keep, h, w, ksize, kept_idx, table, nullptr,
                            stream, "svtad_table_build");
}

extern "C" int svtad_topk_select(const float* scores, int n_seg, int seg_len, int k_keep,
                                 int64_t* idx, void* stream) {
    SV_CHECK_ARG(n_seg == 0 || k_keep == 0 || idx != nullptr, "svtad_topk_select: idx is null");
    return table_build_impl(scores, n_seg, seg_len, k_keep, 0, 0, 0, nullptr, nullptr, idx, stream,
                            "svtad_topk_select");
}

extern "C" int svtad_table_select_remap(const float* scores, const int32_t* table_in, int B, int n_prev,
                                        int k_keep, int kk, int32_t* kept_idx, int64_t* idx, int32_t* table_out,
                                        void* stream) {
    SV_CHECK_ARG(B >= 0 && n_prev > 0 && kk > 0, "svtad_table_select_remap: bad sizes");
    SV_CHECK_ARG(k_keep >= 0 && k_keep <= n_prev, "svtad_table_select_remap: k_keep=%d outside [0, %d]", k_keep, n_prev);
    SV_CHECK_ARG((long)B * n_prev < (1l << 31), "svtad_table_select_remap: row count does not fit int32 indices");
    if (B == 0 || k_keep == 0) return SVTAD_OK;
    SV_CHECK_ARG(scores && table_in && kept_idx && table_out, "svtad_table_select_remap: null pointer");
    if (n_prev > SEG_MAX)
        return set_error(SVTAD_ERR_UNSUPPORTED, "svtad_table_select_remap: n_prev=%d exceeds the %d-token limit", n_prev, SEG_MAX);
    return segment_launch(scores, B, n_prev, k_keep, n_prev, 1, 1, kk, kept_idx, table_out, idx, table_in, (cudaStream_t)stream);
}

extern "C" int svtad_table_remap(const int32_t* table_in, const int64_t* idx, int B, int n_prev,
                                 int n_new, int kk, int32_t* scratch, int32_t* table_out,
                                 void* stream) {
    SV_CHECK_ARG(B >= 0 && n_prev >= 0 && n_new >= 0 && kk > 0, "svtad_table_remap: bad sizes");
    SV_CHECK_ARG((long)B * n_prev < (1l << 31) && (long)B * n_new < (1l << 31),
                 "svtad_table_remap: row count does not fit int32 indices");
    if (B == 0 || n_new == 0) return SVTAD_OK;
    SV_CHECK_ARG(table_in && idx && scratch && table_out, "svtad_table_remap: null pointer");
    cudaStream_t s = (cudaStream_t)stream;
    SV_CUDA(cudaMemsetAsync(scratch, 0xFF, (size_t)B * n_prev * sizeof(int32_t), s));
    long rows = (long)B * n_new;
    remap_scatter_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, s>>>(idx, scratch, B, n_prev, n_new);
    SV_LAUNCH_CHECK("remap_scatter_kernel");
    long total = rows * kk;
    remap_gather_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(table_in, idx, scratch, table_out, B, n_prev, n_new, kk);
    SV_LAUNCH_CHECK("remap_gather_kernel");
    return SVTAD_OK;
}

extern "C" int svtad_table_check(const int32_t* nbr, int64_t n, int kk, int tokens_per_batch,
                                 int32_t* status, void* stream) {
    SV_CHECK_ARG(n >= 0 && kk > 0 && tokens_per_batch >= 0, "svtad_table_check: bad sizes");
    SV_CHECK_ARG(status != nullptr, "svtad_table_check: status is null");
    cudaStream_t s = (cudaStream_t)stream;
    SV_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), s));
    if (n == 0) return SVTAD_OK;
    SV_CHECK_ARG(nbr != nullptr, "svtad_table_check: nbr is null");
    long total = (long)n * kk;
    table_check_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(nbr, (long)n, kk, tokens_per_batch, status);
    SV_LAUNCH_CHECK("table_check_kernel");
    return SVTAD_OK;
}
