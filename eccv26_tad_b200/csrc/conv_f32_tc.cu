// fp32 SparseConv2D on the tensor cores: forward, input gradient (gather form) and weight gradient, every operand split
// into three bf16 values.
//
// An fp32 value is the exact sum of three bf16 ones, x = x1 + x2 + x3 (8 + 8 + 8 bits, each the rounded rest of the ones
// before; the method of G. Henry, P. T. P. Tang and A. Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For
// Higher-Precision Computations", ARITH 2019), and a product needs six of the nine partial products: x1 w1, x1 w2, x2 w1, x1 w3, x2 w2, x3 w1; the three that
// are left out are below 2^-26 of it.  What would spoil the result is the accumulator: tcgen05.mma cuts its sum off towards
// zero at every instruction (measured, relative error of a sum of N(0,1) products against 64 bits: 2.4e-8 after one
// instruction of 16 products, 6.5e-8 after 4, 1.2e-7 after 8, 4.7e-7 after 32, nearly all of it bias).  So a sum stays in
// tensor memory for one step of 64 products only and is then added to the running sum in registers, rounded to nearest; the
// small partial products have columns of their own.  Errors against 64 bits (2-norm) over 4 to 1024 channels, 9 to 49
// taps, 59 to 7 080 rows: forward 5e-8 to 1.4e-7, input gradient 5e-8 to 1.2e-7, weight gradient 5e-8 to 1.4e-7; the
// CUDA-core kernels (conv_f32.cu) 6e-8 to 4.7e-7, 6e-8 to 3.0e-7, 1.2e-7 to 3.6e-7, each call's larger than here.  Values
// are split as 2^16 times what they are, and the sums brought back by 2^-32: the last bit that fp32 has, 2^-149, is then the
// last that bf16 has, and planes lose nothing however small the value is (without it: all of a tensor below 4e-34 made errors
// of 3e-6 at 1e-35, 3e-4 at 1e-37).
//
// A value that is infinite, NaN or above 2^112 makes its planes NaN, also in sums that it has no part in (the rows of a tile
// that lack a neighbor are rows of zeros), and a sum above 2^96 is infinite.  Sums that are not finite are therefore made again from
// the fp32 values, by all warps of the CTA, before they are stored.  us a call of 4 720 rows, C = 192, ordinary values / one
// infinity in each operand / all infinite (a thread per sum: 1 150 and 7 430 with one): forward 27 / 164 / 200, input gradient 27 /
// 152 / 195, weight gradient 25 / 114 / 114; the CUDA-core kernels, whatever the values, 59, 62 and 51.
//
// Measured (graph replays, before: the CUDA-core kernels): 784 rows, C = 192, keep 50 %: forward 21.7 -> 11.0 us, input
// gradient 22.9 -> 11.0; 4 720 rows, C = 192, keep 30 %: 55.0 -> 26.8, 58.0 -> 27.1, weight gradient 49.8 -> 22.0; 5 880
// rows, full grid, 320 -> 96: 144 -> 44, 134 -> 40, 103 -> 57.  What bounds the loops: eight warps that load, split and store
// (900 issue slots per scheduler and step of 1 500 cycles; 768 cycles of tensor work) and the gathered rows' trip from L2, which is
// one step long.
#include <cfloat>

#include "tc_common.cuh"

namespace svtad {

constexpr int T3_A_WARPS = 8;
constexpr int T3_E_WARPS = 4;
constexpr int T3_THREADS = (T3_A_WARPS + 1 + T3_E_WARPS) * 32;      // the MMA warp (TMEM owner) sits between them
constexpr int T3_FW_THREADS = T3_THREADS + 32;         // forward, input gradient: a warp more, for the weights
constexpr int T3_BN = 64;
constexpr int T3_A_PLANE = A_TILE_BYTES, T3_B_PLANE = T3_BN * 128;
constexpr int T3_STAGE = 3 * (T3_A_PLANE + T3_B_PLANE);      // weight gradient
constexpr int T3_RING = 2, T3_B_STAGE = 3 * T3_B_PLANE;      // forward, input gradient: A in tensor memory
constexpr int T3_RAWS = 4, T3_RAW = 64 * T3_BN * 4;          // ... and the weights' fp32 tiles
constexpr int T3_A_COL = 256, T3_A_COLS = 96;               // behind two accumulators of 128 columns
constexpr int T3_COLS = 3 * T3_BN;                     // accumulator columns of a step

typedef unsigned long long t3_pair;                    // two fp32 values
__device__ __forceinline__ t3_pair t3_pack(uint32_t lo, uint32_t hi) {
    t3_pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void t3_unpack(t3_pair v, uint32_t& lo, uint32_t& hi) { asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v)); }
__device__ __forceinline__ t3_pair t3_add(t3_pair a, t3_pair b) {
    t3_pair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ t3_pair t3_mul(t3_pair a, t3_pair b) {
    t3_pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
constexpr t3_pair T3_UP = 0x4780000047800000ull, T3_DOWN = 0x2F8000002F800000ull;      // 2^16 and 2^-32, twice
__device__ __forceinline__ t3_pair t3_neg_add(t3_pair a, t3_pair b) {      // b - a
    t3_pair r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(b), "l"(a));
    return r;
}

// Two values -> the three planes of 2^16 times them, packed, the second with its sign turned: plane minus value is one instruction on the
// half of a packed register.  (Widening the plane by a shift and a mask first: 16.5 cycles per pair and scheduler instead of
// 12.7 in a loop of its own - conversions, shifts, masks and selects go through a pipe of half the width.)
__device__ __forceinline__ void t3_split2(float a, float b, uint32_t (&p)[3]) {
    uint32_t lo, hi;
    t3_unpack(t3_mul(t3_pack(__float_as_uint(a), __float_as_uint(b)), T3_UP), lo, hi);
    a = __uint_as_float(lo);
    b = __uint_as_float(hi);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        p[q] = pack2(a, b, false);
        if (q < 2)
            asm("{\n\t.reg .b16 lo, hi;\n\t"
                "mov.b32 {lo, hi}, %2;\n\t"
                "sub.rn.f32.bf16 %0, lo, %0;\n\t"
                "sub.rn.f32.bf16 %1, hi, %1;\n\t}" : "+f"(a), "+f"(b) : "r"(p[q]));
    }
}
// eight values -> four packed words of each plane
__device__ __forceinline__ void t3_split8(const float (&v)[8], uint32_t (&p)[3][4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        uint32_t w[3];
        t3_split2(v[2 * e], v[2 * e + 1], w);
#pragma unroll
        for (int q = 0; q < 3; ++q) p[q][e] = w[q];
    }
}

// What is read for a row that is not there: an address like any other instead of a branch or a select at the load.  Rows
// of more channels than this are refused by f32_tc_wanted().
constexpr int T3_MOST = 4096;
__device__ __align__(32) float t3_zeros[T3_MOST];

// FULL: all channels are there and 32-byte aligned; else those four for which first / second say so
template <bool FULL>
__device__ __forceinline__ void t3_load8(float (&v)[8], const float* p, bool first, bool second) {
    if constexpr (FULL) {
        asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p));
    } else {
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 a = first ? __ldg(reinterpret_cast<const float4*>(p)) : none, b = second ? __ldg(reinterpret_cast<const float4*>(p) + 1) : none;
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
}
__device__ __forceinline__ void t3_sts16(uint32_t dst, const uint32_t (&v)[4]) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void t3_sts8(uint32_t dst, uint32_t lo, uint32_t hi) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst), "r"(lo), "r"(hi) : "memory");
}
// 16 rows x 32 words of tensor memory: lane t holds words 8 j + 2 (t % 4), + 1 of row t / 4 (v[4 j], v[4 j + 1]) and of row
// t / 4 + 8 (v[4 j + 2], v[4 j + 3])
__device__ __forceinline__ void t3_tmem_st(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
                 ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
                   "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void t3_tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D += A (tensor memory) . B
__device__ __forceinline__ void t3_umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}

// what the warp wrote to a buffer is the tensor core's to read
__device__ __forceinline__ void t3_filled(uint32_t bar, int lane) {
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// A step's instructions, A and B in shared memory and both MN-major: 16 products further are 16 rows of 128 bytes.  Columns
// [0, 64) of the accumulator get x1 w1, [64, 128) x1 w2 + x2 w1, [128, 192) the rest.  The planes w1, w2, w3 lie one behind the
// other, so three instructions do the six products: x1 . [w1 w2 w3] (N = 192), x2 . [w1 w2] (N = 128), x3 . w1 (N = 64), and
// read A three times instead of six (with N = 64 throughout, shared memory would be the bound by a factor of 1.5).
__device__ __forceinline__ void t3_issue(uint32_t d, uint32_t stage) {
    const uint32_t a_lo = ((stage & 0x3FFFFu) >> 4) | smem_desc_lbo_bits(8192);
    const uint32_t b_lo = a_lo + (3 * T3_A_PLANE >> 4);
    constexpr uint32_t hi = smem_desc_hi(1024);
    constexpr uint32_t i3 = make_idesc(1, 1, 1, TILE_M, 3 * T3_BN), i2 = make_idesc(1, 1, 1, TILE_M, 2 * T3_BN), i1 = make_idesc(1, 1, 1, TILE_M, T3_BN);
#pragma unroll
    for (int ks = 0; ks < STAGE_K / 16; ++ks) {
        const uint32_t a = a_lo + ks * 128, b = b_lo + ks * 128;
        umma_f16_lh(d, a, hi, b, hi, i3, ks != 0 ? 1u : 0u);
        umma_f16_lh_acc(d + T3_BN, a + (T3_A_PLANE >> 4), hi, b, hi, i2);
        umma_f16_lh_acc(d + 2 * T3_BN, a + 2 * (T3_A_PLANE >> 4), hi, b, hi, i1);
    }
}
// The same with A in tensor memory (three planes of 32 columns), where the accumulator is left two blocks of 64 columns: x1 w1, and
// all others with their sign turned (the second planes are stored negative).
template <bool B_MN>
__device__ __forceinline__ void t3_issue_ts(uint32_t d, uint32_t a_tmem, uint32_t b_tile) {
    const uint32_t b1 = ((b_tile & 0x3FFFFu) >> 4) | (B_MN ? smem_desc_lbo_bits(8192) : 0u), b2 = b1 + (T3_B_PLANE >> 4), b3 = b2 + (T3_B_PLANE >> 4);
    constexpr uint32_t hi = smem_desc_hi(1024), neg = 1u << 13;
    constexpr uint32_t i2 = make_idesc(1, 0, B_MN, TILE_M, 2 * T3_BN), i1 = make_idesc(1, 0, B_MN, TILE_M, T3_BN);
#pragma unroll
    for (int ks = 0; ks < STAGE_K / 16; ++ks) {
        const uint32_t a = a_tmem + ks * 8, o = ks * (B_MN ? 128 : 2);
        t3_umma_ts(d, a, b1 + o, hi, i2, ks != 0 ? 1u : 0u);                      // x1 w1, -(x1 w2)
        t3_umma_ts(d + T3_BN, a + 32, b1 + o, hi, i1, 1u);                        // -(x2 w1)
        t3_umma_ts(d + T3_BN, a, b3 + o, hi, i1 | neg, 1u);                       // -(x1 w3)
        t3_umma_ts(d + T3_BN, a + 32, b2 + o, hi, i1 | neg, 1u);                  // -(x2 w2)
        t3_umma_ts(d + T3_BN, a + 64, b1 + o, hi, i1 | neg, 1u);                  // -(x3 w1)
    }
}
// a step's accumulator, added to the lane's running sums
template <int BLOCKS>
__device__ __forceinline__ void t3_drain(t3_pair (&sum)[T3_BN / 2], uint32_t t_addr) {
#pragma unroll
    for (int c = 0; c < T3_BN; c += 16) {
        uint32_t g0[16], g1[16], g2[16];
        tmem_ld16(t_addr + c, g0);
        tmem_ld16(t_addr + T3_BN + c, g1);
        if (BLOCKS == 3) tmem_ld16(t_addr + 2 * T3_BN + c, g2);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            t3_pair step = t3_pack(g0[2 * e], g0[2 * e + 1]);
            const t3_pair turned = t3_pack(g1[2 * e], g1[2 * e + 1]);
            if (BLOCKS == 3) step = t3_add(step, t3_neg_add(turned, t3_pack(g2[2 * e], g2[2 * e + 1])));
            else step = t3_neg_add(turned, step);
            sum[c / 2 + e] = t3_add(sum[c / 2 + e], step);
        }
    }
}

__device__ __forceinline__ bool t3_finite(float v) { return fabsf(v) <= FLT_MAX; }
__device__ __forceinline__ bool t3_finite(const float4& v) { return t3_finite(v.x) && t3_finite(v.y) && t3_finite(v.z) && t3_finite(v.w); }

// The values of `rows` rows of the tile from row `lo` on, of 64 columns, that came out infinite or NaN, from the fp32 values: a warp
// per four rows and sixteen columns; lanes l % 4 have four columns each and lanes l / 4 four of 32 channels, whose sums are added up
// at the end.  All threads of the CTA call; out and s_row as they left them.  A function of its own, so that the kernel keeps its
// registers.
template <bool DGRAD>
__device__ __noinline__ void t3_redo(float* out, const float* const* s_row, const float* w, const float* bias, long row0, int lo, int rows,
                                     int n0, long n, int cred, int cn, int cin, int cout, int kk) {
    const int lane = threadIdx.x & 31, items = (rows + 3) / 4 * 4;
    for (int item = threadIdx.x >> 5; item < items; item += T3_FW_THREADS / 32) {
        const int r0 = lo + item / 4 * 4, col = n0 + item % 4 * 16 + (lane & 3) * 4;
        int at[4];
        bool bad = false;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            at[r] = r0 + r < lo + rows && row0 + r0 + r < n ? r0 + r : r0;
            if (r == lane >> 3 && row0 + r0 < n && col < cn) bad = !t3_finite(*reinterpret_cast<const float4*>(out + (row0 + at[r]) * cn + col));
        }
        if (!__any_sync(0xffffffffu, bad)) continue;
        float sum[4][4] = {};
        for (int k = 0; k < kk; ++k) {
            const float* a[4];
            bool there[4], any = false;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                a[r] = s_row[k * TILE_M + at[r]];
                there[r] = a[r] != t3_zeros;
                any = any || there[r];
            }
            if (!any) continue;
            if (col < cn) {
                const float* wk = DGRAD ? w + ((long)(kk - 1 - k) * cin + col) * cout : w + (long)k * cin * cout + col;
#pragma unroll 2
                for (int c = (lane >> 2) * 4; c < cred; c += 32) {
                    float4 av[4], wv[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) av[r] = __ldg(reinterpret_cast<const float4*>(a[r] + c));
#pragma unroll
                    for (int q = 0; q < 4; ++q) wv[q] = __ldg(reinterpret_cast<const float4*>(DGRAD ? wk + (long)q * cout + c : wk + (long)(c + q) * cout));
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        if (!there[r]) continue;           // zeros would make NaN of an infinite weight
                        const float x[4] = {av[r].x, av[r].y, av[r].z, av[r].w};
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                const float4 v = DGRAD ? wv[q] : wv[i];
                                const int c4 = DGRAD ? i : q;
                                sum[r][q] = fmaf(x[i], c4 == 0 ? v.x : c4 == 1 ? v.y : c4 == 2 ? v.z : v.w, sum[r][q]);
                            }
                    }
                }
            }
            // a lane's NaN is one of the whole sum; once all are NaN that is what they stay
            unsigned nans = 0;
#pragma unroll
            for (int e = 0; e < 16; ++e) nans |= (sum[e >> 2][e & 3] != sum[e >> 2][e & 3] ? 1u : 0u) << e;
#pragma unroll
            for (int d = 4; d < 32; d <<= 1) nans |= __shfl_xor_sync(0xffffffffu, nans, d);
            if (__all_sync(0xffffffffu, nans == 0xffffu || col >= cn)) break;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int d = 4; d < 32; d <<= 1) sum[r][q] += __shfl_xor_sync(0xffffffffu, sum[r][q], d);
            if (r != lane >> 2 || row0 + r0 >= n || col >= cn) continue;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float* to = out + (row0 + at[r]) * cn + col + q;
                if (!t3_finite(*to)) *to = sum[r][q] + (!DGRAD && bias != nullptr ? __ldg(bias + col + q) : 0.f);
            }
        }
    }
}

// A walk over a tile's K steps, (tap, 64 channels), the taps ascending; SKIP: those of a mask alone
template <bool SKIP>
struct T3Steps {
    uint64_t left;                         // SKIP: the current tap is the lowest bit
    int k, c0;
    __device__ __forceinline__ T3Steps(uint64_t taps, int st, int chunks) {
        k = st / chunks;
        c0 = (st - k * chunks) * STAGE_K;
        if constexpr (SKIP) {
            left = taps;
            for (; k > 0; --k) left &= left - 1;
            k = __ffsll((long long)left) - 1;
        }
    }
    __device__ __forceinline__ void next(int cred) {
        c0 += STAGE_K;
        if (c0 < cred) return;
        c0 = 0;
        if constexpr (SKIP) {
            left &= left - 1;
            k = __ffsll((long long)left) - 1;
        } else {
            ++k;
        }
    }
};

// ---------------------------------------------------------------------------------------------
// forward / input gradient: a CTA per 128 rows x 64 columns; K steps are (tap, 64 channels)
// ---------------------------------------------------------------------------------------------
// A goes from registers to tensor memory, B through shared memory: with both in shared memory its 128 bytes a cycle were the bound
// (72 KB written, 96 KB read and the loads' way through L1 a step; 4 720 rows, C = 192: 34.2 us instead of 28.8).
// The weights' tiles come as fp32 through TMA, several steps ahead: every CTA reads each of them once, from L2, while most gathered
// rows are found in L1 again by the taps that follow.  Loaded to registers one step ahead they were what the warps waited for:
// 784 rows, C = 192: 12.2 -> 11.1 us, 4 720 rows: 28.8 -> 28.0, input gradient 28.2 -> 26.4, 80 rows, C = 1024: 31.3 -> 25.5.
// SKIP: taps that none of the tile's rows has a neighbor at are left out.  With few rows that may be most of them (8 rows, C = 192,
// four tokens a slice, 7 x 7: 23.4 -> 12.3 us), with more hardly one, and finding out costs 0.25 us and the loop 1 to 2 %: up to 64 rows.
// SPLIT: a cluster of G CTAs shares the tile's K steps; the sums meet in shared memory, in the order of the CTAs.
template <bool DGRAD, bool SPLIT, bool FULL, bool SKIP>
__global__ void __launch_bounds__(T3_FW_THREADS, 1)
conv_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const float* __restrict__ a, const int32_t* __restrict__ nbr, const float* __restrict__ w,
                   const float* __restrict__ bias, float* __restrict__ out, const int32_t* __restrict__ status, long n, int cred,
                   int cn, int cin, int cout, int kk, int tpb, int n_blks, int G, int* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    TmaTail* tail = reinterpret_cast<TmaTail*>(smem + T3_RING * T3_B_STAGE + T3_RAWS * T3_RAW);
    const float** s_row = reinterpret_cast<const float**>(tail + 1);      // [kk][128] gathered rows, or the row of zeros
    volatile int* s_abort = &tail->abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t stage_base = smem_u32(smem), raw_base = stage_base + T3_RING * T3_B_STAGE;
    __shared__ uint64_t s_raw_full[T3_RAWS], s_raw_empty[T3_RAWS];
    __shared__ uint32_t s_taps[2][T3_FW_THREADS / 32];         // SKIP: per warp, the taps of the neighbors it has seen
    const int share = SPLIT ? (int)blockIdx.x % G : 0, item = SPLIT ? (int)blockIdx.x / G : (int)blockIdx.x;
    const long row0 = (long)(item / n_blks) * TILE_M;
    const int n0 = item % n_blks * T3_BN;
    const int chunks = (cred + STAGE_K - 1) / STAGE_K;
    int total = kk * chunks, k_lo = SPLIT ? total * share / G : 0, k_hi = SPLIT ? total * (share + 1) / G : total;

    if (warp == T3_A_WARPS) {
        tmem_alloc(smem_u32(&tail->tmem_slot), 512);
        tmem_relinquish();
    }
    if (tid == T3_A_WARPS * 32) {
        for (int s = 0; s < T3_RING; ++s) {
            mbar_init(smem_u32(&tail->full[s]), T3_A_WARPS);
            mbar_init(smem_u32(&tail->empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&tail->accum_full[b]), 1);
            mbar_init(smem_u32(&tail->accum_empty[b]), T3_E_WARPS * 32);
        }
        for (int r = 0; r < T3_RAWS; ++r) {
            mbar_init(smem_u32(&s_raw_full[r]), 1);
            mbar_init(smem_u32(&s_raw_empty[r]), T3_A_WARPS);
        }
        tail->abort_flag = 0;
        fence_mbar_init();
        tma_prefetch_map(&map_w);
    }
    pdl_wait();
    if (DGRAD && status != nullptr && (__ldg(status) & SVTAD_TABLE_ASYMMETRIC)) {      // uniform over the grid
        __syncthreads();
        if (warp == T3_A_WARPS) tmem_dealloc(tail->tmem_slot, 512);
        return;
    }
    {
        const int32_t* rows = nbr + row0 * kk;
        const int valid = (int)(n - row0 < TILE_M ? n - row0 : TILE_M) * kk;
        uint64_t mine = 0;
        for (int e = tid; e < TILE_M * kk; e += T3_FW_THREADS) {
            const int r = e / kk, k = e - r * kk;
            const int raw = e < valid ? __ldg(rows + e) : -1;
            const long j = (long)raw + (tpb > 0 ? ((row0 + r) / tpb) * (long)tpb : 0);
            const bool there = raw >= 0 && j < n;
            s_row[k * TILE_M + r] = there ? a + j * cred : t3_zeros;
            if (SKIP && there) mine |= 1ull << k;
        }
        if constexpr (SKIP) {
            const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)mine), hi = __reduce_or_sync(0xffffffffu, (uint32_t)(mine >> 32));
            if (lane == 0) {
                s_taps[0][warp] = lo;
                s_taps[1][warp] = hi;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tail->tmem_slot;
    pdl_trigger();
    uint64_t taps = 0;
    if constexpr (SKIP) {
        taps = (uint64_t)__reduce_or_sync(0xffffffffu, lane < T3_FW_THREADS / 32 ? s_taps[1][lane] : 0u) << 32 |
               __reduce_or_sync(0xffffffffu, lane < T3_FW_THREADS / 32 ? s_taps[0][lane] : 0u);
        total = __popcll(taps) * chunks;
        k_lo = SPLIT ? total * share / G : 0;
        k_hi = SPLIT ? total * (share + 1) / G : total;
    }

    t3_pair sum[T3_BN / 2];
    const int q = warp & 3;
    if (warp < T3_A_WARPS) {
        // ------------------------------------------------------------------ producers: all of them fill every buffer
        // A: 16 rows per warp, straight from registers to tensor memory.  A lane loads channels 8 c .. + 7 and 32 + 8 c .. + 7
        // (c = lane % 4) of rows lane / 4 and lane / 4 + 8; its j-th four channels become products 16 j + 4 c .. + 3 of the
        // step, an order that B's rows (forward) or 8-byte pieces of them (input gradient) follow.
        const int c8 = (lane & 3) * 8, r16 = (warp & 3) * 32 + (warp >> 2) * 16 + (lane >> 2);
        const uint32_t a_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32 + (warp >> 2) * 16) << 16) + T3_A_COL;
        // B: rows warp * 8 + {0 .. 3}, + 4, eight columns per lane; the fp32 tile is two boxes of 32 columns.  Eight lanes are half of
        // a row and the other half of its neighbor, a half-warp has four rows: neither the loads nor the stores meet a bank twice.
        const int sub = lane & 7, row4 = ((lane >> 4) + (lane >> 3 & 1) * 2) ^ (sub >> 2), b_row = warp * 8 + row4;
        const uint32_t b_raw = raw_base + (sub >> 2) * (T3_RAW / 2) + b_row * 128 + (((sub & 3) * 2 ^ (b_row & 7)) << 4);
        uint32_t b_place;
        if (DGRAD) {
            b_place = b_row * 128 + ((((sub >> 2) * 4 + (sub >> 1 & 1)) ^ (b_row & 7)) << 4) + (sub & 1) * 8;
        } else {
            const int r = (warp >> 2) * 32 + (warp & 3) * 4 + row4;
            b_place = r * 128 + ((sub ^ (r & 7)) << 4);
        }
        const uint32_t b_next = DGRAD ? 4 * 128 : 16 * 128;       // rows of the second four
        float va[2][2][8];
        T3Steps<SKIP> at(taps, k_lo, chunks);
        const float* const* my_row = s_row + r16;
        auto load_a = [&] {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float* row = my_row[at.k * TILE_M + 8 * r] + at.c0 + c8;
#pragma unroll
                for (int h = 0; h < 2; ++h) t3_load8<FULL>(va[r][h], row + 32 * h, at.c0 + c8 + 32 * h < cred, at.c0 + c8 + 32 * h + 4 < cred);
            }
        };
        if (k_lo < k_hi) load_a();
        int s = 0, rs = 0;
        uint32_t ph = 1, rph = 0;
        for (int st = k_lo; st < k_hi; ++st) {
            uint32_t pa[3][16];
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t p[3][4];
                    t3_split8(va[r][h], p);
#pragma unroll
                    for (int q = 0; q < 3; ++q)
#pragma unroll
                        for (int e = 0; e < 4; ++e) pa[q][8 * h + 4 * (e >> 1) + 2 * r + (e & 1)] = p[q][e];
                }
            // the next step's loads are on their way while this one is multiplied; behind the last step this one's again
            if (st + 1 < k_hi) at.next(cred);
            load_a();
            if (!mbar_wait_warp(smem_u32(&tail->empty[s]), ph, s_abort, err, 81)) break;
            tc_fence_after();
#pragma unroll
            for (int q = 0; q < 3; ++q) t3_tmem_st(a_addr + s * T3_A_COLS + q * 32, pa[q]);
            const uint32_t b_tile = stage_base + s * T3_B_STAGE + b_place;
            if (!mbar_wait_warp(smem_u32(&s_raw_full[rs]), rph, s_abort, err, 89)) break;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // rows b_row and b_row + 4: the second one's chunks lie across the swizzle
                float vb[8];
                const uint32_t src = (b_raw + rs * T3_RAW + h * 512) ^ (h ? 64u : 0u);
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(vb[4 * q]), "=f"(vb[4 * q + 1]), "=f"(vb[4 * q + 2]), "=f"(vb[4 * q + 3]) : "r"(src ^ (q ? 16u : 0u)) : "memory");
                uint32_t p[3][4];
                t3_split8(vb, p);
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const uint32_t dst = b_tile + q * T3_B_PLANE + h * b_next;
                    if (DGRAD) {
                        t3_sts8(dst ^ (h ? 64u : 0u), p[q][0], p[q][1]);
                        t3_sts8(dst ^ (h ? 96u : 32u), p[q][2], p[q][3]);
                    } else {
                        t3_sts16(dst, p[q]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&s_raw_empty[rs]));
            if (++rs == T3_RAWS) { rs = 0; rph ^= 1u; }
            t3_tmem_st_wait();
            tc_fence_before();
            t3_filled(smem_u32(&tail->full[s]), lane);
            if (++s == T3_RING) { s = 0; ph ^= 1u; }
        }
    } else if (warp == T3_A_WARPS) {
        // ------------------------------------------------------------------ MMA issuer (whole warp waits, one lane issues)
        int s = 0;
        uint32_t ph = 0;
        for (int st = 0; st < k_hi - k_lo; ++st) {
            const int buf = st & 1;
            const bool ok = mbar_wait(smem_u32(&tail->accum_empty[buf]), ((st >> 1) & 1) ^ 1, s_abort, err, 82) &&
                            mbar_wait(smem_u32(&tail->full[s]), ph, s_abort, err, 83);
            tc_fence_after();
            if (elect_one_sync()) {
                t3_issue_ts<!DGRAD>(tmem_base + buf * (2 * T3_BN), tmem_base + T3_A_COL + s * T3_A_COLS, stage_base + s * T3_B_STAGE);
                umma_commit(smem_u32(&tail->empty[s]));
                umma_commit(smem_u32(&tail->accum_full[buf]));
            }
            if (!__all_sync(0xffffffffu, ok)) break;
            if (++s == T3_RING) { s = 0; ph ^= 1u; }
        }
    } else if (warp == T3_A_WARPS + 1 + T3_E_WARPS) {
        // ------------------------------------------------------------------ weights: fp32 tiles, T3_RAWS steps ahead
        if (lane == 0) {
            T3Steps<SKIP> at(taps, k_lo, chunks);
            int rs = 0;
            uint32_t ph = 1;
            for (int st = k_lo; st < k_hi; ++st) {
                if (!mbar_wait(smem_u32(&s_raw_empty[rs]), ph, s_abort, err, 90)) break;
                const uint32_t bar = smem_u32(&s_raw_full[rs]), dst = raw_base + rs * T3_RAW;
                mbar_expect_tx(bar, T3_RAW);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    tma_load_3d(dst + h * (T3_RAW / 2), &map_w, (DGRAD ? at.c0 : n0) + 32 * h, DGRAD ? n0 : at.c0, DGRAD ? kk - 1 - at.k : at.k, bar);
                at.next(cred);
                if (++rs == T3_RAWS) { rs = 0; ph ^= 1u; }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ four warps keep the sums
#pragma unroll
        for (int c = 0; c < T3_BN / 2; ++c) sum[c] = 0;
        const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
        for (int st = 0; st < k_hi - k_lo; ++st) {
            const int buf = st & 1;
            if (!mbar_wait_warp(smem_u32(&tail->accum_full[buf]), (st >> 1) & 1, s_abort, err, 84)) break;
            tc_fence_after();
            t3_drain<2>(sum, t_addr + buf * (2 * T3_BN));
            tc_fence_before();
            mbar_arrive(smem_u32(&tail->accum_empty[buf]));
        }
    }
    // The sums go through shared memory, those of a shared tile to the CTA that finishes their rows, so that all threads store whole
    // lines (a lane that stores its own row takes 16 bytes of 32 lines at a time: 4 720 rows, C = 192: 28.0 us instead of 25.7; with
    // the shared sums by rows as well, 784 rows took 11.1 instead of 10.4).  A CTA whose wait gave up stops the whole
    // cluster: the others' sums are not finished with what it left behind.
    __syncthreads();
    if constexpr (SPLIT) {
        if (tid < G && *s_abort) store_to_cta(smem_u32(&tail->abort_flag), tid, 1);
        cluster_barrier();          // every CTA's instructions are done: nothing is left in the rings, which take the sums now
    }
    const bool all = *s_abort == 0;
    const int per = SPLIT ? (TILE_M + G - 1) / G : TILE_M;  // rows that a CTA finishes: [share * per, ...)
    const int pitch = per | 1;                              // [CTA the sums come from][column / 4][row], an odd number of rows apart
    if (all && warp > T3_A_WARPS && warp <= T3_A_WARPS + T3_E_WARPS) {
        const int r = q * 32 + lane, owner = SPLIT ? r / per : 0;
        const uint32_t here = stage_base + (share * (T3_BN / 4) * pitch + r - owner * per) * 16;
        const uint32_t dst = SPLIT ? map_to_cta(here, owner) : here;
#pragma unroll
        for (int c = 0; c < T3_BN / 4; ++c) {
            uint32_t u[4];
            t3_unpack(t3_mul(sum[2 * c], T3_DOWN), u[0], u[1]);
            t3_unpack(t3_mul(sum[2 * c + 1], T3_DOWN), u[2], u[3]);
            if (SPLIT) asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + c * pitch * 16), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]) : "memory");
            else t3_sts16(dst + c * pitch * 16, u);
        }
    }
    if constexpr (SPLIT) cluster_barrier(); else __syncthreads();
    const float4* sums = reinterpret_cast<const float4*>(smem);
    const int rows = !all ? 0 : share * per + per <= TILE_M ? per : TILE_M - share * per;
    bool again = false;
    for (int e = tid; e < rows * (T3_BN / 4); e += T3_FW_THREADS) {
        const int r = e / (T3_BN / 4), c = e % (T3_BN / 4), col = n0 + 4 * c;
        const long row = row0 + share * per + r;
        if (row >= n || col >= cn) continue;
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int p = 0; p < (SPLIT ? G : 1); ++p) {
            const float4 u = sums[(p * (T3_BN / 4) + c) * pitch + r];
            f.x += u.x; f.y += u.y; f.z += u.z; f.w += u.w;
        }
        if (!DGRAD && bias != nullptr) {
            const float4 b = __ldg(reinterpret_cast<const float4*>(bias + col));
            f.x += b.x; f.y += b.y; f.z += b.z; f.w += b.w;
        }
        again = again || !t3_finite(f);
        *reinterpret_cast<float4*>(out + row * cn + col) = f;
    }
    tc_fence_before();
    if (__syncthreads_or(again)) t3_redo<DGRAD>(out, s_row, w, bias, row0, share * per, rows, n0, n, cred, cn, cin, cout, kk);
    settle_after_abort(s_abort);
    if (warp == T3_A_WARPS) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// ---------------------------------------------------------------------------------------------
// weight gradient: D[128 input channels of a tap][64 columns] over the (row, neighbor) pairs that exist, 64 a step
// ---------------------------------------------------------------------------------------------
// A CTA takes a range of tokens, lists the pairs that its tap has there (1.3 of 4 tokens at keep 30 %, against a step for every
// 64 tokens) and works through the list.  The centre tap has every token for a pair, so its tokens are cut into more ranges than
// the others' (a CTA whose list is empty costs little, one whose list is three times as long sets the time).  Both operands lie
// as rows of tokens (MN-major).  Partials to ws_w[range][kk][cin][cout].  The bias gradient's CTAs, behind all others, add up
// gy's columns to ws_b[range][cout].
constexpr int T3_SEG = 4096;               // tokens listed at a time
struct T3Units {
    int m_blks, n_blks, centre;
    int own, others, bias;                 // ranges of tokens for the centre tap, the other taps, the bias gradient (0: not wanted)
};

// Segments of T3_SEG tokens: their pairs (row of gy, row of x), ascending, and behind them (-1, -1) up to a whole step.  Each of the
// first eight warps, all of which call, lists an eighth of it between two barriers of theirs.
__device__ __forceinline__ void t3_list_pairs(int2* s_pair, int* s_count, int* s_pairs, const int32_t* nbr, long seg, long i_end,
                                              long n, int kk, int tap, int tpb) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int Q = T3_SEG / T3_A_WARPS / 32;
    const int len = (int)min((long)T3_SEG, i_end - seg), eighth = (len + 255) / 256 * 32;
    int jj[Q], cnt = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int at = warp * eighth + q * 32 + lane;
        jj[q] = q * 32 < eighth && at < len ? __ldg(nbr + (seg + at) * kk + tap) : -1;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const long i = seg + warp * eighth + q * 32 + lane, j = (long)jj[q] + (tpb > 0 ? (i / tpb) * (long)tpb : 0);
        jj[q] = jj[q] >= 0 && j < n ? (int)j : -1;
        cnt += __popc(__ballot_sync(0xffffffffu, jj[q] >= 0));
    }
    if (lane == 0) s_count[warp] = cnt;
    named_bar_sync(1, T3_A_WARPS * 32);         // also: nobody reads the last segment's list any more
    int at = 0, pairs = 0;
#pragma unroll
    for (int q = 0; q < T3_A_WARPS; ++q) {
        at += q < warp ? s_count[q] : 0;
        pairs += s_count[q];
    }
    if (tid == 0) *s_pairs = pairs;
    if (tid < STAGE_K && pairs + tid < (pairs + STAGE_K - 1) / STAGE_K * STAGE_K) s_pair[pairs + tid] = make_int2(-1, -1);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const unsigned m = __ballot_sync(0xffffffffu, jj[q] >= 0);
        if (jj[q] >= 0) s_pair[at + __popc(m & ((1u << lane) - 1u))] = make_int2((int)(seg + warp * eighth + q * 32 + lane), jj[q]);
        at += __popc(m);
    }
    named_bar_sync(1, T3_A_WARPS * 32);
}

// The tile's sums [column / 4][row] that came out infinite or NaN, from the fp32 values of the pairs, ascending, eight rows by four
// columns per thread of the first eight warps, all of which call.  A function of its own, so that the kernel keeps its registers.
__device__ __noinline__ void t3_redo_wgrad(float* sums, int2* s_pair, int* s_count, int* s_pairs, const float* gy, const float* x,
                                           const int32_t* nbr, long i_begin, long i_end, long n, int m0, int n0, int cin, int cout,
                                           int kk, int tap, int tpb) {
    const int r0 = (threadIdx.x >> 4) * 8, c = threadIdx.x & 15, ci = m0 + r0, co = n0 + 4 * c;
    const bool g_there = co < cout, lo_there = ci < cin, hi_there = ci + 4 < cin;
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    float acc[8][4] = {};
    for (long seg = i_begin; seg < i_end; seg += T3_SEG) {
        t3_list_pairs(s_pair, s_count, s_pairs, nbr, seg, i_end, n, kk, tap, tpb);
        const int pairs = *s_pairs;
#pragma unroll 4
        for (int p = 0; p < pairs; ++p) {
            const int2 ij = s_pair[p];
            const float4* xr = reinterpret_cast<const float4*>(x + (long)ij.y * cin + ci);
            const float4 g = g_there ? __ldg(reinterpret_cast<const float4*>(gy + (long)ij.x * cout + co)) : none;
            const float4 lo = lo_there ? __ldg(xr) : none, hi = hi_there ? __ldg(xr + 1) : none;
            const float xv[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                acc[r][0] = fmaf(xv[r], g.x, acc[r][0]);
                acc[r][1] = fmaf(xv[r], g.y, acc[r][1]);
                acc[r][2] = fmaf(xv[r], g.z, acc[r][2]);
                acc[r][3] = fmaf(xv[r], g.w, acc[r][3]);
            }
        }
    }
    sums += (c * (TILE_M + 1) + r0) * 4;
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (!t3_finite(sums[r * 4 + q])) sums[r * 4 + q] = acc[r][q];
}

template <bool FULL>
__global__ void __launch_bounds__(T3_THREADS, 1)
wgrad_f32_tc_kernel(const float* __restrict__ gy, const float* __restrict__ x, const int32_t* __restrict__ nbr,
                    float* __restrict__ ws_w, float* __restrict__ ws_b, long n, int cin, int cout, int kk, int tpb, T3Units u,
                    int* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    TmaTail* tail = reinterpret_cast<TmaTail*>(smem + T3_RING * T3_STAGE);
    int2* s_pair = reinterpret_cast<int2*>(tail + 1);      // [T3_SEG] the pairs: row of gy, row of x
    __shared__ int s_count[T3_A_WARPS], s_pairs, s_end;      // s_end: number of steps, once known
    volatile int* s_abort = &tail->abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t stage_base = smem_u32(smem);

    // which (tap, blocks, range)
    const int tiles = u.m_blks * u.n_blks, own_units = tiles * u.own, all_units = own_units + (kk - 1) * tiles * u.others;
    int tap, tile, range, ranges;
    if ((int)blockIdx.x < own_units) {
        tap = u.centre; ranges = u.own;
        tile = blockIdx.x / ranges; range = blockIdx.x - tile * ranges;
    } else if ((int)blockIdx.x < all_units) {
        const int b = blockIdx.x - own_units;
        ranges = u.others;
        tile = b / ranges; range = b - tile * ranges;
        tap = tile / tiles; tile -= tap * tiles;
        if (tap >= u.centre) ++tap;
    } else {
        const int b = blockIdx.x - all_units;
        ranges = u.bias;
        tile = b / ranges; range = b - tile * ranges;
        tap = kk;
    }
    const int m0 = tap < kk ? tile / u.n_blks * TILE_M : 0, n0 = (tap < kk ? tile % u.n_blks : tile) * T3_BN;
    const long each = (n + ranges - 1) / ranges, i_begin = min(n, range * each), i_end = min(n, i_begin + each);

    if (tap == kk) {
        // column sums of gy: four columns and every 16th row per thread in two chains, the 32 sums added in pairs
        pdl_wait();
        pdl_trigger();
        const int by = tid >> 4, col = n0 + (tid & 15) * 4;
        float4* part = reinterpret_cast<float4*>(smem);     // [16][16]
        auto add = [](float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; };
        if (by < 16) {
            float4 sum[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll 2
            for (long i = i_begin + by; i < i_end; i += 32) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (col < cout && i + 16 * h < i_end) add(sum[h], __ldg(reinterpret_cast<const float4*>(gy + (i + 16 * h) * cout + col)));
            }
            add(sum[0], sum[1]);
            part[tid] = sum[0];
        }
#pragma unroll
        for (int d = 8; d > 0; d >>= 1) {
            __syncthreads();
            if (by < d) add(part[tid], part[tid + d * 16]);
        }
        if (by == 0 && col < cout) *reinterpret_cast<float4*>(ws_b + (long)range * cout + col) = part[tid];
        return;
    }

    if (warp == T3_A_WARPS) {
        tmem_alloc(smem_u32(&tail->tmem_slot), 512);
        tmem_relinquish();
    }
    if (tid == T3_A_WARPS * 32) {
        for (int s = 0; s < T3_RING; ++s) {
            mbar_init(smem_u32(&tail->full[s]), T3_A_WARPS);
            mbar_init(smem_u32(&tail->empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&tail->accum_full[b]), 1);
            mbar_init(smem_u32(&tail->accum_empty[b]), T3_E_WARPS * 32);
        }
        tail->abort_flag = 0;
        fence_mbar_init();
    }
    // producers: the first half of the warps fills the first 64 channels of A, the others the second; eight lanes per row,
    // eight channels each
    constexpr int A_ITS = TILE_M / T3_A_WARPS / 4, B_ITS = STAGE_K / T3_A_WARPS / 4;
    const int sub8 = (lane & 7) * 8, rg = lane >> 3;
    const int half = warp / (T3_A_WARPS / 2), a_tok = warp % (T3_A_WARPS / 2) * (A_ITS * 4), b_tok = warp * (B_ITS * 4);
    const int ca = m0 + half * 64 + sub8, cb = n0 + sub8;
    const bool real = m0 + half * 64 < cin;                // else zeros, written once
    if (warp < T3_A_WARPS && !real) {
        for (int s = 0; s < T3_RING; ++s)
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int c = 0; c < A_ITS; ++c)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(stage_base + s * T3_STAGE + p * T3_A_PLANE + warp * (A_ITS * 512) + c * 512 + lane * 16), "r"(0) : "memory");
        fence_proxy_async();
    }
    if (tid == 0) s_end = 0x7fffffff;
    pdl_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tail->tmem_slot;
    pdl_trigger();

    bool again = false;
    if (warp < T3_A_WARPS) {
        // ------------------------------------------------------------------ producers: all of them fill every buffer
        const uint32_t place[2] = {(uint32_t)(rg * 128 + (((lane & 7) ^ rg) << 4)), (uint32_t)((4 + rg) * 128 + (((lane & 7) ^ (4 + rg)) << 4))};
        float v[A_ITS + B_ITS][8];
        auto store = [&](uint32_t rows, uint32_t plane, int it, const float (&f)[8]) {
            uint32_t p[3][4];
            t3_split8(f, p);
#pragma unroll
            for (int q = 0; q < 3; ++q) t3_sts16(rows + (it >> 1) * 1024 + place[it & 1] + q * plane, p[q]);
        };
        auto load = [&](int st, int it) {
            if (it < A_ITS) {
                const int j = s_pair[st * STAGE_K + a_tok + 4 * it + rg].y;
                t3_load8<FULL>(v[it], j >= 0 ? x + (long)j * cin + ca : t3_zeros + sub8, ca < cin, ca + 4 < cin);
            } else {
                const int i = s_pair[st * STAGE_K + b_tok + 4 * (it - A_ITS) + rg].x;
                t3_load8<FULL>(v[it], i >= 0 ? gy + (long)i * cout + cb : t3_zeros + sub8, cb < cout, cb + 4 < cout);
            }
        };
        bool alive = true;
        int s = 0, done = 0;
        uint32_t ph = 1;
        // A warp whose wait gave up goes on taking part in every segment's two barriers, as the others may not know of it yet.
        for (long seg = i_begin; seg < i_end; seg += T3_SEG) {
            t3_list_pairs(s_pair, s_count, &s_pairs, nbr, seg, i_end, n, kk, tap, tpb);
            if (!alive) continue;
            const int steps = (s_pairs + STAGE_K - 1) / STAGE_K;
            if (steps > 0) {
#pragma unroll
                for (int it = 0; it < A_ITS + B_ITS; ++it)
                    if (it >= A_ITS || real) load(0, it);
            }
            for (int st = 0; st < steps; ++st) {
                if (!mbar_wait_warp(smem_u32(&tail->empty[s]), ph, s_abort, err, 85)) { alive = false; break; }
                const uint32_t a_rows = stage_base + s * T3_STAGE + warp * (A_ITS * 512), b_rows = stage_base + s * T3_STAGE + 3 * T3_A_PLANE + b_tok * 128;
                const int next = st + 1 < steps ? st + 1 : st;
                if (real) {
#pragma unroll
                    for (int it = 0; it < A_ITS; ++it) {
                        store(a_rows, T3_A_PLANE, it, v[it]);
                        load(next, it);
                    }
                }
#pragma unroll
                for (int it = A_ITS; it < A_ITS + B_ITS; ++it) {
                    store(b_rows, T3_B_PLANE, it - A_ITS, v[it]);
                    load(next, it);
                }
                t3_filled(smem_u32(&tail->full[s]), lane);
                if (++s == T3_RING) { s = 0; ph ^= 1u; }
            }
            done += steps;
        }
        // one more round, which carries nothing: the end
        if (alive && mbar_wait_warp(smem_u32(&tail->empty[s]), ph, s_abort, err, 85)) {
            if (tid == 0) s_end = done;
            t3_filled(smem_u32(&tail->full[s]), lane);
        }
    } else if (warp == T3_A_WARPS) {
        // ------------------------------------------------------------------ MMA issuer (whole warp waits, one lane issues)
        for (int g = 0;; ++g) {
            const int s = g % T3_RING, buf = g & 1;
            const bool ok = mbar_wait(smem_u32(&tail->accum_empty[buf]), ((g >> 1) & 1) ^ 1, s_abort, err, 86) &&
                            mbar_wait(smem_u32(&tail->full[s]), g / T3_RING & 1, s_abort, err, 87);
            const bool end = *reinterpret_cast<volatile int*>(&s_end) == g;
            __syncwarp();
            tc_fence_after();
            if (elect_one_sync()) {
                if (!end) {
                    t3_issue(tmem_base + buf * T3_COLS, stage_base + s * T3_STAGE);
                    umma_commit(smem_u32(&tail->empty[s]));
                }
                umma_commit(smem_u32(&tail->accum_full[buf]));
            }
            if (!__all_sync(0xffffffffu, ok && !end)) break;
        }
    } else {
        // ------------------------------------------------------------------ the last four warps keep the sums
        t3_pair sum[T3_BN / 2];
#pragma unroll
        for (int c = 0; c < T3_BN / 2; ++c) sum[c] = 0;
        const uint32_t t_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        for (int g = 0;; ++g) {
            const int buf = g & 1;
            if (!mbar_wait_warp(smem_u32(&tail->accum_full[buf]), (g >> 1) & 1, s_abort, err, 88)) break;
            if (*reinterpret_cast<volatile int*>(&s_end) == g) break;
            tc_fence_after();
            t3_drain<3>(sum, t_addr + buf * T3_COLS);
            tc_fence_before();
            mbar_arrive(smem_u32(&tail->accum_empty[buf]));
        }
        // the sums leave through the ring, which nothing is in any more, as the forward's do
        const uint32_t dst = stage_base + ((warp & 3) * 32 + lane) * 16;
#pragma unroll
        for (int c = 0; c < T3_BN / 4; ++c) {
            uint32_t f[4];
            t3_unpack(t3_mul(sum[2 * c], T3_DOWN), f[0], f[1]);
            t3_unpack(t3_mul(sum[2 * c + 1], T3_DOWN), f[2], f[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) again = again || !t3_finite(__uint_as_float(f[e]));
            t3_sts16(dst + c * (TILE_M + 1) * 16, f);
        }
    }
    if (__syncthreads_or(again) && *s_abort == 0) {
        if (warp < T3_A_WARPS)
            t3_redo_wgrad(reinterpret_cast<float*>(smem), s_pair, s_count, &s_pairs, gy, x, nbr, i_begin, i_end, n, m0, n0, cin, cout, kk, tap, tpb);
        __syncthreads();
    }
    if (*s_abort == 0) {
        const float4* sums = reinterpret_cast<const float4*>(smem);
        float* to = ws_w + (((long)range * kk + tap) * cin + m0) * cout + n0;
        for (int e = tid; e < TILE_M * (T3_BN / 4); e += T3_THREADS) {
            const int r = e / (T3_BN / 4), c = e % (T3_BN / 4);
            if (m0 + r < cin && n0 + 4 * c < cout) *reinterpret_cast<float4*>(to + (long)r * cout + 4 * c) = sums[c * (TILE_M + 1) + r];
        }
    }
    tc_fence_before();
    __syncthreads();
    settle_after_abort(s_abort);
    if (warp == T3_A_WARPS) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// fixed-order sum of the ranges' partials, four elements per thread; the bias gradient behind the weights
__global__ void __launch_bounds__(128)
wgrad_f32_tc_sum_kernel(const float* __restrict__ ws_w, const float* __restrict__ ws_b, T3Units u, float* __restrict__ gw,
                        float* __restrict__ gb, int cin, int cout, int kk) {
    pdl_wait();
    pdl_trigger();
    const long n_w = (long)kk * cin * cout;
    long e = (blockIdx.x * 128l + threadIdx.x) * 4;
    const float* src = ws_w;
    float* dst = gw;
    long stride = n_w;
    int ranges = u.bias;
    if (e >= n_w) {
        e -= n_w;
        if (gb == nullptr || e >= cout) return;
        src = ws_b; dst = gb; stride = cout;
    } else {
        ranges = e / ((long)cin * cout) == u.centre ? u.own : u.others;
    }
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int q = 0; q < ranges; ++q) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(src + q * stride + e));
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    *reinterpret_cast<float4*>(dst + e) = s;
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
// whole blocks of 64 channels, rows that 32-byte loads may read
static bool t3_full(int cin, int cout, const void* a, const void* b) {
    return cin % STAGE_K == 0 && cout % STAGE_K == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 31) == 0;
}

template <bool DGRAD, bool SPLIT, bool FULL, bool SKIP>
static int launch_f32_tc(const ConvArgs& p, const int32_t* status, int G, cudaStream_t s) {
    const int cn = DGRAD ? p.cin : p.cout, cred = DGRAD ? p.cout : p.cin;
    const size_t table = (size_t)p.kk * TILE_M * sizeof(float*);
    const int n_blks = (cn + T3_BN - 1) / T3_BN;
    const long tiles = (p.n + TILE_M - 1) / TILE_M * n_blks;
    const size_t smem = 1024 + T3_RING * T3_B_STAGE + T3_RAWS * T3_RAW + sizeof(TmaTail) + table;
    auto kern = conv_f32_tc_kernel<DGRAD, SPLIT, FULL, SKIP>;
    int rc = tc_ensure_smem(reinterpret_cast<const void*>(kern), smem);
    if (rc) return rc;
    CUtensorMap map_w;
    const uint64_t dims[3] = {(uint64_t)p.cout, (uint64_t)p.cin, (uint64_t)p.kk};
    const uint32_t box[3] = {32, 64, 1};
    rc = tc_make_map_sw(&map_w, 3, p.w, dims, box, TC_MAP_F32, 128);
    if (rc) return rc;
    SV_CUDA(launch_pdl(kern, dim3((unsigned)(tiles * G)), dim3(T3_FW_THREADS), smem, s, SPLIT ? G : 1, map_w, (const float*)p.a, p.nbr,
                       (const float*)p.w, (const float*)p.bias, (float*)p.out, status, (long)p.n, cred, cn, p.cin, p.cout, p.kk, p.tpb,
                       n_blks, G, tc_error_ptr()));
    return SVTAD_OK;
}

template <bool DGRAD>
static int dispatch_f32_tc(const ConvArgs& p, const int32_t* status, cudaStream_t s) {
    const int cn = DGRAD ? p.cin : p.cout, cred = DGRAD ? p.cout : p.cin;
    const long tiles = (p.n + TILE_M - 1) / TILE_M * ((cn + T3_BN - 1) / T3_BN), sms = tc_num_sms();
    const int steps = p.kk * ((cred + STAGE_K - 1) / STAGE_K);
    // a step takes 0.72 us and sharing a tile out 2.5; clusters of three and more do not pack a GPC's SMs completely
    const int sizes[6] = {2, 3, 4, 5, 6, 8}, limit[6] = {148, 132, 128, 125, 126, 112};
    double best = (double)((tiles + sms - 1) / sms) * steps * 0.72;
    int G = 1;
    for (int g = 0; g < 6; ++g) {
        if (tiles * sizes[g] * 148 > limit[g] * sms) continue;
        const double u = (steps + sizes[g] - 1) / sizes[g] * 0.72 + 2.5;
        if (u < best) { best = u; G = sizes[g]; }
    }
    const bool full = t3_full(p.cin, p.cout, p.a, p.w);
    if (G == 1) return full ? launch_f32_tc<DGRAD, false, true, false>(p, status, 1, s) : launch_f32_tc<DGRAD, false, false, false>(p, status, 1, s);
    if (p.n <= 64) return full ? launch_f32_tc<DGRAD, true, true, true>(p, status, G, s) : launch_f32_tc<DGRAD, true, false, true>(p, status, G, s);
    return full ? launch_f32_tc<DGRAD, true, true, false>(p, status, G, s) : launch_f32_tc<DGRAD, true, false, false>(p, status, G, s);
}

// Where these kernels take over from those on the CUDA cores, us there and here.  Forward and input gradient from four rows on: 1
// row, C = 192, 3 x 3: 6.2 and 6.9; 8 rows, one neighbor in nine / five / all: 6.4 and 7.1 / 10.1 and 8.9 / 10.7 and 9.7; 96 rows, C = 512:
// 32.2 and 13.6 at one in four, 39.5 and 14.1 at all.  (Above 64 rows a table in which hardly a row has any neighbor is the exception: 96
// rows, C = 512, none: 10.1 and 13.8; so are sparse tables over at most 32 channels, half of a step: 16 000 rows, 32 -> 192, density
// 0.14: 27.5 and 34.9, 0.42: 38.9 and 35.7, 0.96: 70.5 and 36.0.)
// The weight gradient has 7 us per CTA whatever it holds, one CTA an SM, and cuts its tokens for one pair in three tokens.  So it
// loses where there is little to do, mostly on full tables (64 -> 64, 3 x 3, density 0.15 / 0.95: 1 100 rows 9.8 and 9.5 / 9.8 and
// 12.9, 2 400 rows 12.4 and 11.3 / 15.1 and 14.8), and where many CTAs have few pairs each, as with wide
// stencils (density 0.15: 800 rows, C = 512, 5 x 5: 64 and 66, 7 x 7: 105 and 125; 1 100 rows: 85 and 70, 140 and 133; at density 0.3 it
// wins at 640; C = 1024, 3 x 3, 640 rows, density 0.2 / 0.4: 91 and 96 / 131 and 109).
bool f32_tc_wanted(int op, int64_t n, int cin, int cout, int kk) {
    if (cin > T3_MOST || cout > T3_MOST) return false;
    if (op != SVTAD_OP_WGRAD) return n >= 4 || (n > 0 && kk == 1);
    const double work = (double)n * kk * ((cin + 63) / 64 * 64) * ((cout + 63) / 64 * 64);
    const long ctas = (long)kk * ((cin + TILE_M - 1) / TILE_M) * ((cout + T3_BN - 1) / T3_BN);
    return n >= (kk > 9 && ctas > 600 ? 900 : 640) && (n >= 2600 || work >= 7e7);
}

int f32_tc_fwd(const ConvArgs& p, cudaStream_t s) { return dispatch_f32_tc<false>(p, nullptr, s); }
int f32_tc_dgrad(const ConvArgs& p, const int32_t* status, cudaStream_t s) { return dispatch_f32_tc<true>(p, status, s); }

// at most `limit` ranges of tokens (what the workspace of the kernels without tensor cores holds the partials of)
int f32_tc_wgrad(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n, int cin, int cout, int kk, int tpb,
                 float* ws_w, float* ws_b, int limit, cudaStream_t s) {
    T3Units u{(cin + TILE_M - 1) / TILE_M, (cout + T3_BN - 1) / T3_BN, kk / 2, 1, 1, 0};
    const long tiles = (long)u.m_blks * u.n_blks, sms = tc_num_sms();
    // one in three tokens is assumed to have a pair; a step takes 0.9 us, a CTA 7 besides, the partials go through L2 twice
    double best = 0;
    for (int c = 1; c <= limit; ++c) {
        const int own = 3 * c < limit ? 3 * c : limit;
        const long ctas = tiles * ((kk - 1) * c + own);
        const double steps = n * 0.33 / c > (double)n / own ? n * 0.33 / c : (double)n / own;
        const double t = (double)((ctas + sms - 1) / sms) * (steps / STAGE_K * 0.9 + 7) + ((double)c * (kk - 1) + own) * cin * cout * 8 / 6e6;
        if (c == 1 || t < best * 0.98) { best = t; u.others = c; u.own = own; }
    }
    if (gb != nullptr) u.bias = limit < 16 ? limit : 16;
    const size_t smem = 1024 + T3_RING * T3_STAGE + sizeof(TmaTail) + T3_SEG * sizeof(int2);
    auto kern = t3_full(cin, cout, x, gy) ? wgrad_f32_tc_kernel<true> : wgrad_f32_tc_kernel<false>;
    int rc = tc_ensure_smem(reinterpret_cast<const void*>(kern), smem);
    if (rc) return rc;
    const long ctas = tiles * ((kk - 1) * u.others + u.own) + (long)u.n_blks * u.bias;
    SV_CUDA(launch_pdl(kern, dim3((unsigned)ctas), dim3(T3_THREADS), smem, s, 1, (const float*)gy, (const float*)x, nbr, ws_w, ws_b, (long)n,
                       cin, cout, kk, tpb, u, tc_error_ptr()));
    const long quads = ((long)kk * cin * cout + (gb ? cout : 0)) / 4;
    SV_CUDA(launch_pdl(wgrad_f32_tc_sum_kernel, dim3((unsigned)((quads + 127) / 128)), dim3(128), 0, s, 1, ws_w, ws_b, u, (float*)gw,
                       (float*)gb, cin, cout, kk));
    return SVTAD_OK;
}

}  // namespace svtad
