// Weight gradient over the pairs of a table's plan: tcgen05 / TMEM, 16-bit tensors, fp32 accumulate.
//
//   gw[k] = sum over the pairs (i, j) of tap k of x[j]^T . gy[i]
//
// The kernel without a plan (wgrad_hybrid_kernel) walks all tokens for every tap and multiplies zero rows where a
// neighbor is pruned; here a tap's reduction runs over its list, 64 pairs per step: a third of the steps at keep 30 %,
// a quarter with a 5x5 stencil.  Work unit = (tap, 128 input channels, BN output channels), and one more row of units,
// fed with ones instead of x and walking all rows, for the column sums of gy: the bias gradient.  The list lengths are
// on the device and very uneven (the centre tap has every row for a pair), so the units are laid end to end and each
// persistent CTA takes an equal run of steps, whatever units it cuts: whole units are rounded and stored directly, the
// cut ones leave their fp32 pieces, at most two per CTA, to a second launch that adds them up in a fixed order.  (Whole
// units dealt out in turn left a quarter of the SMs' time idle.)  A unit's accumulator is drained while the next unit's
// main loop fills the other one.
//
// Both operands are gathered rows in the MN-major 128-byte-swizzled layout (64 tokens x 64 channels = 8 KB blocks), so a
// step of 128 x 256 copies 48 KB; what bounds the loop is the SM's path to L2 (48 KB in ~ 700 cycles against 512 cycles
// of tensor work).
#include <cstdlib>

#include "plan.cuh"
#include "tc_common.cuh"

namespace svtad {

// Two warps fill a buffer, 32 of its 64 tokens each.  A warp gets a 512-byte cp.async out every 40 cycles or so however
// many bytes are in flight (measured: 25 / 49 / 70 bytes per cycle and SM with 2 / 4 / 8 warps), so with four producers
// a step of 48 KB took 1 780 cycles.
constexpr int WP_A_WARPS = 8, WP_PER_BUF = 2, WP_GROUPS = WP_A_WARPS / WP_PER_BUF;
constexpr int WP_THREADS = (WP_A_WARPS + 5) * 32;      // then the MMA warp (TMEM owner) and four epilogue warps
constexpr int WP_MAX_KK = 49;
constexpr int WP_MIN_RUN = 20;             // steps that pay for a CTA's start and its piece's trip through memory
// MH = 128-channel halves of x that a unit takes: 2 where the input channels come in blocks of 256.  Then gy's rows are
// gathered once for both: 32 KB per 512 cycles of tensor work instead of 48 KB, at the price of the second accumulator (the
// two fill the tensor memory, so a unit is drained before the next one starts).  A step is 64 / MH pairs.
template <int MH> constexpr int wp_step() { return STAGE_K / MH; }
constexpr int WP_TURN_BYTES = 4 * 2 * 32 * 64;         // per epilogue warp two chunks of 32 rows x 32 values, turned on their way out

struct WgradUnits {
    int m_blks, n_blks;                    // blocks of x (128 * MH channels) and of gy (BN channels)
    int step;                              // pairs per step
    int taps, bias;                        // bias: whether the bias gradient is asked for
    int runs;                              // CTAs of the main launch
};

// the units' lengths and places in the end-to-end order, from the lists' lengths; made by every block (all threads call)
struct UnitMap {
    int len[WP_MAX_KK + 1];                // steps of a unit of the tap; [taps]: bias units
    long base[WP_MAX_KK + 2];              // first step of the tap's units
    int runs;                              // of about equal length, none below MIN_RUN steps
    long run_len, run_rest;

    __device__ void make(const WgradUnits& u, const PlanView& plan, long n) {
        const int t = threadIdx.x;
        if (t <= u.taps) len[t] = (int)(((t < u.taps ? (long)__ldg(plan.count + t) : u.bias ? n : 0) + u.step - 1) / u.step);
        __syncthreads();
        if (t <= u.taps + 1) {
            long at = 0;
            for (int k = 0; k < t; ++k) at += (long)len[k] * (k < u.taps ? u.m_blks * u.n_blks : u.n_blks);
            base[t] = at;
            if (t == u.taps + 1) {
                runs = (int)(at / WP_MIN_RUN < 1 ? 1 : at / WP_MIN_RUN < u.runs ? at / WP_MIN_RUN : u.runs);
                run_len = at / runs;
                run_rest = at - run_len * runs;
            }
        }
        __syncthreads();
    }
    // the boundary behind a run: (tap, unit, pieces of the unit) where it is the first one inside a unit, else no pieces
    __device__ int4 cut(const WgradUnits& u, int run) const {
        if (run + 1 >= runs) return make_int4(0, 0, 0, 0);
        const long cut = run_begin(run + 1);
        int tap, unit, step, parts = 2;
        at(u, cut, tap, unit, step);
        if (step == 0 || cut - step < run_begin(run)) return make_int4(0, 0, 0, 0);
        while (run + parts < runs && run_begin(run + parts) < cut - step + len[tap]) ++parts;
        return make_int4(tap, unit, parts, 0);
    }
    // first step of a run; runs behind the last one are empty
    __device__ long run_begin(int run) const { return run >= runs ? run_len * runs + run_rest : run * run_len + (run < run_rest ? run : run_rest); }
    // the unit that step `pos` belongs to
    __device__ void at(const WgradUnits& u, long pos, int& tap, int& unit, int& step) const {
        int k = 0;
        while (pos >= base[k + 1]) ++k;    // pos < total
        const int off = (int)(pos - base[k]);
        tap = k;
        unit = off / len[k];
        step = off - unit * len[k];
    }
};

template <int BN, int MH>
__global__ void __launch_bounds__(WP_THREADS, 1)
wgrad_pairs_kernel(const uint16_t* __restrict__ gy, const uint16_t* __restrict__ x, PlanView plan, void* __restrict__ gw,
                   void* __restrict__ gb, float* __restrict__ pieces, int4* __restrict__ cuts, long n, int cin, int cout, WgradUnits units, int nstage,
                   int fp16, int out32, int* __restrict__ err) {
    constexpr int SK = wp_step<MH>(), BLK = SK * 128;       // a block: SK tokens x 64 channels
    constexpr int A_BYTES = 2 * MH * BLK, STAGE_BYTES = A_BYTES + BN / 64 * BLK;
    constexpr int WT = SK / WP_PER_BUF, ITS = WT / 4;       // tokens of a step per warp; copies per lane and block
    constexpr int NBUF = MH == 1 ? 2 : 1;                   // accumulators
    constexpr int TM_COLS = tmem_cols2_for(BN);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    TmaTail* tail = reinterpret_cast<TmaTail*>(smem + (size_t)nstage * STAGE_BYTES + WP_TURN_BYTES);
    __shared__ UnitMap map;
    volatile int* s_abort = &tail->abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t stage_base = smem_u32(smem);

    if (warp == WP_A_WARPS) {
        tmem_alloc(smem_u32(&tail->tmem_slot), TM_COLS);
        tmem_relinquish();
    }
    if (tid == 0) {
        for (int s = 0; s < nstage; ++s) {
            mbar_init(smem_u32(&tail->full[s]), 32 * WP_PER_BUF);      // the copies of the warps that fill it
            mbar_init(smem_u32(&tail->empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&tail->accum_full[b]), 1);
            mbar_init(smem_u32(&tail->accum_empty[b]), 128);
        }
        tail->abort_flag = 0;
        fence_mbar_init();
    }
    tc_fence_before();
    pdl_wait();
    map.make(units, plan, n);
    tc_fence_after();
    const uint32_t tmem_base = tail->tmem_slot;
    pdl_trigger();

    // the CTA's run of steps, piece by piece: steps [s0, s1) of a unit
    long pos = map.run_begin(blockIdx.x);
    const long run_end = map.run_begin(blockIdx.x + 1);
    int tap, m, nb, s0, s1;
    auto next_piece = [&] {
        if (pos >= run_end) return false;
        int unit;
        map.at(units, pos, tap, unit, s0);
        m = tap < units.taps ? unit / units.n_blks : 0;
        nb = unit - m * units.n_blks;
        s1 = (int)(run_end - pos < map.len[tap] - s0 ? s0 + (run_end - pos) : map.len[tap]);
        pos += s1 - s0;
        return true;
    };

    if (warp < WP_A_WARPS) {
        // ------------------------------------------------------------------ producers: two warps per step, groups in turn
        const int sub = lane & 7, rg = lane >> 3;
        const int grp = warp / WP_PER_BUF, part = warp % WP_PER_BUF;
        const int n_prod = nstage < WP_GROUPS ? nstage : WP_GROUPS;      // never more groups than buffers (see the forward kernel)
        bool alive = true;
        int it0 = 0;
        // the lane's place in the buffers: token itr * 4 + rg of the warp's WT, 16-byte chunk sub of each 64-channel block
        const uint32_t lane_dst[2] = {(uint32_t)(part * WT * 128 + rg * 128 + ((sub ^ rg) << 4)), (uint32_t)(part * WT * 128 + rg * 128 + ((sub ^ (4 | rg)) << 4))};
        while (alive && grp < n_prod && next_piece()) {
            const bool ones = tap == units.taps;
            const int count = ones ? (int)n : __ldg(plan.count + tap), steps = s1 - s0;
            const int32_t* li = plan.pair_i + (long)tap * n + s0 * SK;
            const int32_t* lj = plan.pair_j + (long)tap * n + s0 * SK;
            const int left = count - s0 * SK;
            // nothing is read behind the channels of a partial block
            const uint16_t* xa = x + m * (128 * MH) + sub * 8;
            const uint16_t* gb0 = gy + nb * BN + sub * 8;
            const int x_left = cin - (m * (128 * MH) + sub * 8), g_left = cout - (nb * BN + sub * 8);
            int st = ((grp - it0) % n_prod + n_prod) % n_prod;
            int s = (it0 + st) % nstage;
            uint32_t ph = (((it0 + st) / nstage) & 1) ^ 1;
            it0 += steps;
            int vi, vj;
            auto entries = [&](int step) {                 // this lane's pair of a coming step
                const int p = step * SK + part * WT + lane;
                const bool in = step < steps && p < left && lane < WT;
                vi = in ? (ones ? s0 * SK + p : __ldg(li + p)) : -1;
                vj = in && !ones ? __ldg(lj + p) : -1;
            };
            entries(st);
            for (; st < steps; st += n_prod) {
                int ri[ITS], rj[ITS];                       // the rows this lane's copies take
#pragma unroll
                for (int itr = 0; itr < ITS; ++itr) {
                    ri[itr] = __shfl_sync(0xffffffffu, vi, itr * 4 + rg);
                    rj[itr] = __shfl_sync(0xffffffffu, vj, itr * 4 + rg);
                }
                entries(st + n_prod);
                int ok = 1;
                if (lane == 0) ok = mbar_wait(smem_u32(&tail->empty[s]), ph, s_abort, err, 61) ? 1 : 0;
                if (!__shfl_sync(0xffffffffu, ok, 0)) { alive = false; break; }
                __syncwarp();
                const uint32_t a_tile = stage_base + (uint32_t)s * STAGE_BYTES;
                const uint32_t bar = smem_u32(&tail->full[s]);
                if (ones) {
                    const uint32_t one = fp16 ? 0x3C003C00u : 0x3F803F80u;
                    for (int c = lane; c < A_BYTES / WP_PER_BUF / 16; c += 32)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(a_tile + (part * (A_BYTES / WP_PER_BUF / 16) + c) * 16), "r"(one) : "memory");
                    fence_proxy_async();
                } else if (x_left > (2 * MH - 1) * 64) {
#pragma unroll
                    for (int itr = 0; itr < ITS; ++itr) {
                        const int j = rj[itr];
                        const uint16_t* src = static_cast<const uint16_t*>(row_at(xa, j, (uint32_t)cin * 2));
                        const uint32_t dst = a_tile + lane_dst[itr & 1] + itr * 512, bytes = j < 0 ? 0u : 16u;
#pragma unroll
                        for (int b = 0; b < 2 * MH; ++b) cp_async16(dst + b * BLK, src + b * 64, bytes);
                    }
                } else {
#pragma unroll
                    for (int itr = 0; itr < ITS; ++itr) {
                        const int j = rj[itr];
                        const uint32_t dst = a_tile + lane_dst[itr & 1] + itr * 512;
#pragma unroll
                        for (int b = 0; b < 2 * MH; ++b) {
                            const bool there = j >= 0 && x_left > b * 64;
                            cp_async16(dst + b * BLK, there ? xa + (long)j * cin + b * 64 : x, there ? 16u : 0u);
                        }
                    }
                }
#pragma unroll
                for (int itr = 0; itr < ITS; ++itr) {
                    const int i = ri[itr];
                    const uint32_t dst = a_tile + A_BYTES + lane_dst[itr & 1] + itr * 512, bytes = i < 0 ? 0u : 16u;
                    const uint16_t* src = static_cast<const uint16_t*>(row_at(gb0, i, (uint32_t)cout * 2));
                    if (g_left > BN - 64) {
#pragma unroll
                        for (int b = 0; b < BN / 64; ++b) cp_async16(dst + b * BLK, src + b * 64, bytes);
                    } else {
#pragma unroll
                        for (int b = 0; b < BN / 64; ++b) cp_async16(dst + b * BLK, g_left > b * 64 ? src + b * 64 : gy, g_left > b * 64 ? bytes : 0u);
                    }
                }
                cp_async_arrive_noinc(bar);
                s += n_prod;
                while (s >= nstage) { s -= nstage; ph ^= 1u; }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == WP_A_WARPS) {
        // ------------------------------------------------------------------ MMA issuer (whole warp waits, one lane issues)
        const uint32_t idesc = make_idesc(fp16 ? 0 : 1, 1, 1, TILE_M, BN);
        bool alive = true;
        int s = 0;
        uint32_t ph = 0;
        for (int local = 0; next_piece(); ++local) {
            const int buf = local % NBUF, steps = s1 - s0;
            if (!mbar_wait_warp(smem_u32(&tail->accum_empty[buf]), ((local / NBUF) & 1) ^ 1, s_abort, err, 62)) break;
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + buf * BN;
            for (int st = 0; st < steps; ++st) {
                const bool ok = mbar_wait(smem_u32(&tail->full[s]), ph, s_abort, err, 63);
                fence_proxy_async();       // cp.async (generic proxy) writes -> tcgen05.mma (async proxy) reads
                tc_fence_after();
                const uint32_t a_tile = stage_base + (uint32_t)s * STAGE_BYTES;
                if (elect_one_sync()) {
                    // both operands MN-major: 16 tokens per instruction = 2048 B, 64-channel blocks BLK bytes apart
                    const uint32_t a_lo = ((a_tile & 0x3FFFFu) >> 4) | smem_desc_lbo_bits(BLK);
                    const uint32_t b_lo = a_lo + (A_BYTES >> 4);
#pragma unroll
                    for (int h = 0; h < MH; ++h) {
                        const uint32_t ah = a_lo + h * (2 * BLK >> 4);
                        umma_f16_lh(d_tmem + h * BN, ah, smem_desc_hi(1024), b_lo, smem_desc_hi(1024), idesc, st != 0 ? 1u : 0u);
#pragma unroll
                        for (int ks = 1; ks < SK / 16; ++ks)
                            umma_f16_lh_acc(d_tmem + h * BN, ah + ks * 128, smem_desc_hi(1024), b_lo + ks * 128, smem_desc_hi(1024), idesc);
                    }
                    umma_commit(smem_u32(&tail->empty[s]));
                }
                if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
                if (++s == nstage) { s = 0; ph ^= 1u; }
            }
            if (!alive) break;
            if (elect_one_sync()) umma_commit(smem_u32(&tail->accum_full[buf]));
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ epilogue (the last four warps)
        constexpr int NC = BN / 32;
        const int q = warp & 3;
        uint4* turns = reinterpret_cast<uint4*>(smem + (size_t)nstage * STAGE_BYTES) + q * 256;
        if (q == 0 && lane == 0) cuts[blockIdx.x] = map.cut(units, blockIdx.x);
        for (int local = 0; next_piece(); ++local) {
            const int buf = local % NBUF;
            int ok = 1;
            if (lane == 0) ok = mbar_wait(smem_u32(&tail->accum_full[buf]), (local / NBUF) & 1, s_abort, err, 64) ? 1 : 0;
            if (!__shfl_sync(0xffffffffu, ok, 0)) break;
            __syncwarp();
            tc_fence_after();
#pragma unroll 1
            for (int h = 0; h < MH; ++h) {
                const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + (buf + h) * BN;
                const int row = h * 128 + q * 32 + lane, ci = m * (128 * MH) + row, n0 = nb * BN;
                const bool bias = tap == units.taps;
                const int rows = bias ? 1 : cin - (ci - lane);      // of this warp
                // a whole unit goes to the gradient, a piece of a cut one to its place: 0 begins inside a unit, 1 ends there.
                // A store takes as many cycles as it touches lines, and a lane holds a row.  So pieces are kept as
                // [column / 4][row][4], 512 bytes in one run per store, and a whole unit's chunks go through shared memory: a
                // store then writes 64 bytes of each of 8 rows.  (Stored row by row, a piece of 256 x 256 took 9 us to leave.)
                float* part = nullptr;
                if (s0 > 0 || s1 < map.len[tap])
                    part = pieces + (((long)blockIdx.x * 2 + (s0 > 0 ? 0 : 1)) * BN / 4 * (TILE_M * MH) + row) * 4;
                const long at = ((long)tap * cin + (ci - lane)) * cout + n0;      // the warp's first row
                uint32_t va[32], vb[32];
                tmem_ld32(t_addr, va);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    uint32_t (&v)[32] = (c & 1) ? vb : va;
                    tmem_ld_wait();
                    if (c + 1 < NC) tmem_ld32(t_addr + (c + 1) * 32, (c & 1) ? va : vb);
                    if (n0 + c * 32 >= cout) continue;
                    if (part != nullptr) {
                        if (lane < rows) {
#pragma unroll
                            for (int g = 0; g < 8; ++g)
                                *reinterpret_cast<uint4*>(part + (c * 8 + g) * (TILE_M * MH * 4)) = make_uint4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
                        }
                        continue;
                    }
                    uint32_t o[16];
#pragma unroll
                    for (int g = 0; g < 16; ++g) o[g] = pack2(__uint_as_float(v[2 * g]), __uint_as_float(v[2 * g + 1]), fp16 != 0);
                    if (bias) {
                        if (row == 0) {
#pragma unroll
                            for (int g = 0; g < 8; ++g) store_quad(gb, n0 + c * 32 + g * 4, o[2 * g], o[2 * g + 1], fp16 != 0, out32 != 0);
                        }
                        continue;
                    }
                    uint4* turn = turns + (c & 1) * 128;
#pragma unroll
                    for (int g = 0; g < 4; ++g)
                        turn[lane * 4 + (g ^ ((lane >> 1) & 3))] = make_uint4(o[4 * g], o[4 * g + 1], o[4 * g + 2], o[4 * g + 3]);
                    __syncwarp();
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const int r = g * 8 + (lane >> 2);
                        const uint4 t = turn[r * 4 + ((lane & 3) ^ ((r >> 1) & 3))];
                        const long to = at + (long)r * cout + c * 32 + (lane & 3) * 8;
                        if (r >= rows) continue;
                        if (out32) {
                            store_quad(gw, to, t.x, t.y, fp16 != 0, true);
                            store_quad(gw, to + 4, t.z, t.w, fp16 != 0, true);
                        } else {
                            *reinterpret_cast<uint4*>(static_cast<uint16_t*>(gw) + to) = t;
                        }
                    }
                }
                __syncwarp();      // the next half turns its chunks in the same place
            }
            tc_fence_before();
            mbar_arrive(smem_u32(&tail->accum_empty[buf]));
        }
    }
    tc_fence_before();
    __syncthreads();
    settle_after_abort(s_abort);
    if (warp == WP_A_WARPS) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, TM_COLS);
    }
}

// The cut units: grid.x = the boundaries between the runs; the first boundary inside a unit adds its pieces up in the
// order of the runs, with one rounding.  A warp takes 32 rows x 16 columns, a lane a row, so it reads runs of 512 bytes and
// writes sectors; grid.y shares a unit's strips out.  Blocks behind the boundaries clear the gradient of taps that have no
// pair at all.  A boundary's unit comes from the main kernel: with every block looking for its own, this kernel took 25 us
// where it takes 14 now (18 880 rows, C = 256, 5 x 5 taps: 45 MB of pieces).
constexpr int WP_SUM_BLOCKS = 16;
template <int BN, int MH>
__global__ void __launch_bounds__(256, 3)
wgrad_pairs_sum_kernel(const float* __restrict__ pieces, const int4* __restrict__ cuts, PlanView plan, void* __restrict__ gw,
                       void* __restrict__ gb, int cin, int cout, WgradUnits units, int fp16, int out32) {
    pdl_wait();
    pdl_trigger();
    if ((int)blockIdx.x >= units.runs - 1) {
        const int tap = (int)blockIdx.x - (units.runs - 1);
        if (__ldg(plan.count + tap) > 0) return;
        const long plane = (long)cin * cout;
        for (long e = (blockIdx.y * 256l + threadIdx.x) * 4; e < plane; e += gridDim.y * 1024l)
            store_quad(gw, tap * plane + e, 0u, 0u, fp16 != 0, out32 != 0);
        return;
    }
    const int run = (int)blockIdx.x;
    const int4 cut = __ldcg(cuts + run);
    const int tap = cut.x, unit = cut.y, parts = cut.z;
    if (parts == 0) return;
    const int m = tap < units.taps ? unit / units.n_blks : 0, nb = unit - m * units.n_blks;
    const bool bias = tap == units.taps;
    constexpr int ROWS = TILE_M * MH, PIECE = 2 * ROWS * BN;       // a run's two pieces
    for (int strip = blockIdx.y * 8 + (threadIdx.x >> 5); strip < ROWS / 32 * (BN / 16); strip += gridDim.y * 8) {
        const int row = strip % (ROWS / 32) * 32 + (threadIdx.x & 31), col = strip / (ROWS / 32) * 16;
        const int co = nb * BN + col;
        if (co >= cout || (bias ? row > 0 : m * ROWS + row >= cin)) continue;
        // the first run ends in this unit (its second place), the others begin in it
        const float* src = pieces + (long)run * PIECE + (col * ROWS + row * 4);
        float4 sum[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) sum[g] = __ldcg(reinterpret_cast<const float4*>(src + ROWS * BN + g * ROWS * 4));
#pragma unroll 2
        for (int r = 1; r < parts; ++r) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const float4 v = __ldcg(reinterpret_cast<const float4*>(src + (long)r * PIECE + g * ROWS * 4));
                sum[g].x += v.x; sum[g].y += v.y; sum[g].z += v.z; sum[g].w += v.w;
            }
        }
        const long at = (bias ? 0 : ((long)tap * cin + m * ROWS + row) * cout) + co;
#pragma unroll
        for (int g = 0; g < 4; ++g)
            store_quad(bias ? gb : gw, at + g * 4, pack2(sum[g].x, sum[g].y, fp16 != 0), pack2(sum[g].z, sum[g].w, fp16 != 0), fp16 != 0,
                       out32 != 0);
    }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
// blocks of 256 input channels where they leave no more than an eighth of padding (18 880 rows, C = 1024, 3 x 3 taps: 193 -> 133 us
// with the pieces' layout; C = 256, 5 x 5: 53 -> 41 us)
static int pairs_halves(int cin) { return (cin + 255) / 256 * 256 * 8 <= cin * 9 ? 2 : 1; }

// Column block of the weight gradient by pairs: blocks times what a step takes at that width, which goes nearly by the width with
// 128 input channels a block (a step's time as a share of 256 columns': 0.38, 0.49, 0.74 at 64, 128, 192 columns) and less so with 256
// (0.5, 0.675, 0.77); a narrower block from 3 % on.  With the other kernels' step times, 0.55, 0.67, 0.81, a width of 640 went in three
// blocks of 256 instead of five of 128, and 960 in four of 256 instead of five of 192.  us with its sum kernel, C = 640: 14 160 rows,
// density 0.35: 109 and 77; 26 550: 159 and 123; C = 896, 14 160 rows: 163 and 125; C = 960 (256 input channels a block): 148 and 128.
static int pairs_bn(int cin, int cout) {
    if (getenv("SVTAD_TC_BN") != nullptr) return tc_widest_bn(cout);
    const int width[4] = {256, 192, 128, 64};
    const double share[2][4] = {{1.0, 0.74, 0.49, 0.38}, {1.0, 0.77, 0.675, 0.5}};
    int bn = 0;
    double least = 1e30;
    for (int i = 0; i < 4; ++i) {
        const double t = (cout + width[i] - 1) / width[i] * share[pairs_halves(cin) - 1][i];
        if (t < 0.97 * least) { least = t; bn = width[i]; }
    }
    return bn;
}

// per run two pieces and the boundary behind it
size_t pairs_wgrad_ws_bytes(int cin, int cout) {
    const size_t run = 2 * TILE_M * pairs_halves(cin) * pairs_bn(cin, cout) * sizeof(float) + sizeof(int4);
    return (tc_num_sms() * run + 255) / 256 * 256;
}

// Worth it where the lists' third of the steps outweighs gathering gy's rows as well and padding the input channels to
// blocks of 128 (C = 192 loses a quarter of each MMA).
bool pairs_wgrad_wanted(int cin, int kk) { return kk >= 2 && (cin + 127) / 128 * 128 * 4 <= cin * 5; }

template <int BN, int MH>
static int launch_pairs(const void* gy, const void* x, const PlanView& plan, void* gw, void* gb, float* pieces, int64_t n, int cin,
                        int cout, int kk, int fp16, int out32, cudaStream_t s) {
    const WgradUnits u{(cin + 128 * MH - 1) / (128 * MH), (cout + BN - 1) / BN, wp_step<MH>(), kk, gb != nullptr ? 1 : 0, tc_num_sms()};
    const size_t stage = (size_t)wp_step<MH>() * 128 * (2 * MH + BN / 64);
    int nstage = (int)((TC_SMEM_LIMIT - 1024 - sizeof(TmaTail) - sizeof(UnitMap) - 64 - WP_TURN_BYTES) / stage);
    if (nstage > 8) nstage = 8;
    const size_t smem = 1024 + nstage * stage + WP_TURN_BYTES + sizeof(TmaTail);
    auto kern = wgrad_pairs_kernel<BN, MH>;
    int rc = tc_ensure_smem(reinterpret_cast<const void*>(kern), smem);
    if (rc) return rc;
    int4* cuts = reinterpret_cast<int4*>(pieces + (size_t)u.runs * 2 * TILE_M * MH * BN);
    SV_CUDA(launch_pdl(kern, dim3((unsigned)u.runs), dim3(WP_THREADS), smem, s, 1, (const uint16_t*)gy, (const uint16_t*)x, plan, gw, gb,
                      pieces, cuts, (long)n, cin, cout, u, nstage, fp16, out32, tc_error_ptr()));
    SV_CUDA(launch_pdl(wgrad_pairs_sum_kernel<BN, MH>, dim3((unsigned)(u.runs - 1 + kk), WP_SUM_BLOCKS), dim3(256), 0, s, 1, pieces, cuts,
                       plan, gw, gb, cin, cout, u, fp16, out32));
    return SVTAD_OK;
}

int pairs_wgrad(const void* gy, const void* x, const void* plan, void* gw, void* gb, int64_t n, int cin, int cout, int kk,
                int dtype, int grad_dtype, void* ws, size_t ws_bytes, cudaStream_t s) {
    const size_t need = pairs_wgrad_ws_bytes(cin, cout);
    if (ws_bytes < need) return set_error(SVTAD_ERR_WORKSPACE, "svtad_conv_wgrad: workspace %zu < %zu bytes", ws_bytes, need);
    PlanView view;
    plan_layout(n, kk, plan, &view);
    const int fp16 = dtype == SVTAD_F16, out32 = grad_dtype == SVTAD_F32;
    float* pieces = static_cast<float*>(ws);
    auto go = [&](auto one, auto two) {
        return (pairs_halves(cin) == 2 ? two : one)(gy, x, view, gw, gb, pieces, n, cin, cout, kk, fp16, out32, s);
    };
    switch (pairs_bn(cin, cout)) {
        case 64: return go(launch_pairs<64, 1>, launch_pairs<64, 2>);
        case 128: return go(launch_pairs<128, 1>, launch_pairs<128, 2>);
        case 192: return go(launch_pairs<192, 1>, launch_pairs<192, 2>);
        default: return go(launch_pairs<256, 1>, launch_pairs<256, 2>);
    }
}

}  // namespace svtad
