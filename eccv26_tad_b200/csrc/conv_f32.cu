// fp32 SparseConv2D on the CUDA cores: forward, input gradient (gather form) and weight gradient.  The tensor-core kernels
// (conv_f32_tc.cu) take over where f32_tc_wanted() says so; SVTAD_FORCE_PATH=simt keeps everything here.
//
// fp32 tensors cannot go through the tensor cores as TF32 without losing the 1e-5 the reference's fp32 path holds
// (opentad/models/bricks/2d_sparse_v3.cu:545-651, a 32 x 32 shared-memory tile kernel with two __syncthreads per
// 32-deep step; for C_in >= 128 implicit_gemm_v2.cu:197-300, gather + cuBLAS SGEMM + reduce; backward by atomics,
// 2d_sparse_v3.cu:656-745).  What bounds these kernels is the FP32 FMA pipe (72 TFLOP/s measured on a B200), so the work
// is done for pairs only: a (row, tap) whose neighbor is pruned takes no part in a sum.  With tokens kept at random 1.7 /
// 3.1 / 4.9 of 9 taps are there at keep 10 / 30 / 55 %, and hardly any 64-row tile can skip a tap as a whole.
//
//   forward / dgrad   A CTA owns a row tile x 64 columns.  The tile's table is compacted per tap into lists of (row,
//                     neighbor); a list is worked through in blocks of at most 64 pairs, each a small dense product
//                     [pairs x C] . [C x 64] in registers (8 pairs x 4 columns per thread at most, exactly
//                     ceil(pairs / 8) rows of threads' work), added to the tile's sums in shared memory.  A pair's
//                     row occurs once per tap, so there are no conflicts and no atomics, and the sums are made in
//                     ascending tap order.
//   wgrad             A CTA owns 64 x 64 channels of one tap and a range of tokens, compacts the range's pairs and sums
//                     x^T . gy over them; fixed-order reduction over the ranges.  Extra CTAs of the same launch sum gy's
//                     columns for the bias gradient.
//
// Operands travel through a two-stage cp.async ring of 32-deep steps.
#include <atomic>

#include "common.cuh"

namespace svtad {

constexpr int F_BK = 32;
constexpr int F_STAGES = 2;               // three gained nothing and cost a CTA per SM
constexpr int F_MAX_KK = 49;
constexpr int F_BN = 64;                  // columns of a tile
constexpr int F_PAIRS = 64;               // pairs of a block
constexpr int F_THREADS = 128;            // 16 along the columns x 8 along the pairs, up to 8 pairs x 4 columns each
constexpr int F_OSTR = F_BN + 4;          // row stride of the tile's sums

// two fp32 FMAs in one instruction: half the issue slots of the same work, which is what leaves room for the
// shared-memory reads and the loop around them
typedef unsigned long long f2;
__device__ __forceinline__ void f2_fma(f2& d, f2 a, f2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ f2 f2_pack(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }

__device__ __forceinline__ void f_cp16(uint32_t dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t f_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void f_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---------------------------------------------------------------------------------------------------------
// forward / input gradient
// ---------------------------------------------------------------------------------------------------------
struct FwdRing {
    // rows of 32 channels: 16-byte chunk c of row r sits at chunk c ^ (r & 7), so that neither the copies nor the reads
    // of eight neighbouring rows meet in a bank
    float a[F_STAGES][F_PAIRS * F_BK];        // gathered rows: [pair][channel]
    float b[F_STAGES][F_BK * F_BN];           // forward: [channel][column], dgrad: [column][channel] (swizzled as well)
};

// A thread's sums: pairs ty + 8 * i.  Forward: acc[i][q] holds columns tx * 4 + 2 * q and the next; the gathered value is
// doubled in a register.  dgrad, whose weight rows lie along the channels: acc[i][q] holds column tx + 16 * q, its even
// and odd channels apart; nothing has to be doubled.
template <bool DGRAD> struct FAcc { f2 v[8][DGRAD ? 4 : 2]; };

// one 32-deep step of a block with R rows of thread work
template <int R, bool DGRAD>
__device__ __forceinline__ void f_step(FAcc<DGRAD>& acc, const float* as, const float* bs, int tx, int ty) {
#pragma unroll 4
    for (int c4 = 0; c4 < F_BK; c4 += 4) {
        ulonglong2 av[R];                               // four channels as two pairs
#pragma unroll
        for (int i = 0; i < R; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(as + (ty + 8 * i) * F_BK + (((c4 >> 2) ^ ty) << 2));
        if constexpr (DGRAD) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bs + (tx + 16 * q) * F_BK + (((c4 >> 2) ^ (tx & 7)) << 2));
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    f2_fma(acc.v[i][q], av[i].x, b.x);
                    f2_fma(acc.v[i][q], av[i].y, b.y);
                }
            }
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bs + (c4 + c) * F_BN + tx * 4);
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    float lo, hi;
                    f2_unpack(c < 2 ? av[i].x : av[i].y, lo, hi);
                    const float a1 = c & 1 ? hi : lo;
                    const f2 a = f2_pack(a1, a1);
                    f2_fma(acc.v[i][0], a, b.x);
                    f2_fma(acc.v[i][1], a, b.y);
                }
            }
        }
    }
}

// G = CTAs of a cluster that share a tile (1 to 8): each takes an equal share of the tile's steps (weighted by their
// pairs) and the partial tiles are summed through distributed shared memory, CTA 0 first.  bm = rows of a tile, a
// multiple of 32 up to 128.
template <bool DGRAD>
__global__ void __launch_bounds__(F_THREADS)
conv_f32_kernel(const float* __restrict__ x, const int32_t* __restrict__ nbr, const float* __restrict__ w,
                const float* __restrict__ bias, float* __restrict__ out, const int32_t* __restrict__ status, long n,
                int cred, int cn, int cin, int cout, int kk, int tpb, int tiles_n, int bm, int G) {
    if (DGRAD && status != nullptr && (__ldg(status) & SVTAD_TABLE_ASYMMETRIC)) return;     // uniform over the grid
    extern __shared__ __align__(16) unsigned char f_smem_raw[];
    FwdRing& ring = *reinterpret_cast<FwdRing*>(f_smem_raw);
    float* s_out = reinterpret_cast<float*>(&ring + 1);                 // [bm][OSTR]
    int* s_j = reinterpret_cast<int*>(s_out + bm * F_OSTR);             // [kk][bm] gathered rows, compacted per tap
    uint8_t* s_row = reinterpret_cast<uint8_t*>(s_j + kk * bm);         // [kk][bm] the tile rows they belong to
    __shared__ int s_cnt[F_MAX_KK];
    __shared__ int s_item[4 * F_MAX_KK], s_cost[4 * F_MAX_KK];           // item = tap << 16 | first pair << 8 | pairs
    __shared__ int s_first, s_first_c, s_steps;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = tid & 15, ty = tid >> 4;
    const int tile = blockIdx.x / G, grp = blockIdx.x % G;
    const long row0 = (long)(tile / tiles_n) * bm;
    const int n0 = (tile % tiles_n) * F_BN;

    // ---- the tile's table rows, in one trip to memory, to where the ring will be
    int* s_raw = reinterpret_cast<int*>(f_smem_raw);
    {
        const int rows = (int)(n - row0 < bm ? n - row0 : bm), valid = rows * kk * 4;
        const char* src = reinterpret_cast<const char*>(nbr + row0 * kk);
        const uint32_t dst = f_smem(s_raw);
        for (int c = tid * 16; c < valid; c += F_THREADS * 16) f_cp16(dst + c, src + c, min(16, valid - c));
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int e = tid; e < bm * (F_OSTR / 4); e += F_THREADS) reinterpret_cast<float4*>(s_out)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // ---- its pairs: a warp lists every fourth tap, rows ascending
    for (int k = warp; k < kk; k += F_THREADS / 32) {
        int cnt = 0;
        for (int q = 0; q < bm; q += 32) {
            const long i = row0 + q + lane;
            const int raw = i < n ? s_raw[(q + lane) * kk + k] : -1;
            const long j = (long)raw + (tpb > 0 ? (i / tpb) * (long)tpb : 0);
            const bool there = raw >= 0 && j < n;                       // anything out of range reads as zero
            const unsigned m = __ballot_sync(0xffffffffu, there);
            if (there) {
                const int at = k * bm + cnt + __popc(m & ((1u << lane) - 1u));
                s_j[at] = (int)j;
                s_row[at] = (uint8_t)(q + lane);
            }
            cnt += __popc(m);
        }
        if (lane == 0) s_cnt[k] = cnt;
    }
    __syncthreads();
    const int chunks = (cred + F_BK - 1) / F_BK;
    if (warp == 0) {
        // blocks of the lists: as many as needed, equally long (multiples of eight pairs); a block costs its rows of
        // thread work per step
        int items = 0, total = 0;
        for (int k0 = 0; k0 < kk; k0 += 32) {
            const int k = k0 + lane, c = k < kk ? s_cnt[k] : 0;
            const int want = (c + F_PAIRS - 1) / F_PAIRS, each = want > 0 ? ((c + want - 1) / want + 7) & ~7 : 1;
            const int blocks = (c + each - 1) / each, rest = c - (blocks - 1) * each;
            const int cost = blocks > 0 ? (blocks - 1) * (each >> 3) + ((rest + 7) >> 3) : 0;
            int both = blocks | cost << 16;                             // inclusive sums of both over the lanes
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, both, d);
                if (lane >= d) both += t;
            }
            const int i0 = items + (both & 0xffff) - blocks, c0 = total + (both >> 16) - cost;
            for (int q = 0; q < blocks; ++q) {
                s_item[i0 + q] = k << 16 | q * each << 8 | (q + 1 < blocks ? each : rest);
                s_cost[i0 + q] = c0 + q * (each >> 3);
            }
            items += __shfl_sync(0xffffffffu, both & 0xffff, 31);
            total += __shfl_sync(0xffffffffu, both >> 16, 31);
        }
        __syncwarp();
        // this CTA's share: the steps whose start falls into [grp, grp + 1) / G of the total cost
        const int lo = (int)((long)total * chunks * grp / G), hi = (int)((long)total * chunks * (grp + 1) / G);
        int steps = 0;
        unsigned first = 0xffffffffu;
        for (int i = lane; i < items; i += 32) {
            const int r = ((s_item[i] & 255) + 7) >> 3, at = s_cost[i] * chunks;
            const int c_lo = lo <= at ? 0 : min(chunks, (lo - at + r - 1) / r), c_hi = hi <= at ? 0 : min(chunks, (hi - at + r - 1) / r);
            if (c_hi > c_lo) first = min(first, (unsigned)(i << 16 | c_lo));
            steps += c_hi - c_lo;
        }
        steps = __reduce_add_sync(0xffffffffu, steps);
        first = __reduce_min_sync(0xffffffffu, first);
        if (lane == 0) { s_first = first >> 16; s_first_c = first & 0xffff; s_steps = steps; }
    }
    __syncthreads();
    const int steps = s_steps;

    int ld_i = s_first, ld_c = s_first_c;                               // loader's position: item, chunk
    // what a thread copies of a weight tile: 16-byte chunks of its rows - channel rows of F_BN columns in the forward,
    // column rows of 32 channels in dgrad
    constexpr int B_CH = DGRAD ? F_BK / 4 : F_BN / 4, B_ITS = F_BK * F_BN / 4 / F_THREADS;
    auto load_stage = [&](int stage) {
        const int it = s_item[ld_i], k = it >> 16, p0 = (it >> 8) & 255, len = it & 255, r8 = (len + 7) & ~7;
        const int c0 = ld_c * F_BK;
        const uint32_t a_base = f_smem(ring.a[stage]), b_base = f_smem(ring.b[stage]);
        for (int g = tid; g < r8 * (F_BK / 4); g += F_THREADS) {
            const int r = g >> 3, c = c0 + (g & 7) * 4;
            const bool ok = r < len && c < cred;
            const int j = r < len ? s_j[k * bm + p0 + r] : 0;
            f_cp16(a_base + (r * F_BK + (((g ^ r) & 7) << 2)) * 4, ok ? x + (long)j * cred + c : x, ok ? 16u : 0u);
        }
        const float* src = w + (DGRAD ? ((long)(kk - 1 - k) * cin + n0) * cout + c0 : ((long)k * cin + c0) * cout + n0);
        const int r_lim = DGRAD ? cn - n0 : cred - c0, c_lim = DGRAD ? cred - c0 : cn - n0;
#pragma unroll
        for (int q = 0; q < B_ITS; ++q) {
            const int g = tid + q * F_THREADS, r = g / B_CH, ch = g % B_CH;
            const bool ok = r < r_lim && ch * 4 < c_lim;
            f_cp16(b_base + (DGRAD ? r * F_BK + (((ch ^ r) & 7) << 2) : r * F_BN + ch * 4) * 4,
                   ok ? src + r * cout + ch * 4 : w, ok ? 16u : 0u);
        }
        if (++ld_c == chunks) { ld_c = 0; ++ld_i; }
    };

    FAcc<DGRAD> acc;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < (DGRAD ? 4 : 2); ++j) acc.v[i][j] = 0;
#pragma unroll
    for (int s = 0; s < F_STAGES - 1; ++s) {
        if (s < steps) load_stage(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int it_i = s_first, it_c = s_first_c, stage = 0;
    for (int st = 0; st < steps; ++st) {
        asm volatile("cp.async.wait_group %0;" ::"n"(F_STAGES - 2) : "memory");
        __syncthreads();          // step st has landed for every thread; the buffer refilled below is no longer read
        if (st + F_STAGES - 1 < steps) load_stage(stage == 0 ? F_STAGES - 1 : stage - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const int it = s_item[it_i], len = it & 255;
        const float* as = ring.a[stage];
        const float* bs = ring.b[stage];
        switch ((len + 7) >> 3) {
            case 1: f_step<1, DGRAD>(acc, as, bs, tx, ty); break;
            case 2: f_step<2, DGRAD>(acc, as, bs, tx, ty); break;
            case 3: f_step<3, DGRAD>(acc, as, bs, tx, ty); break;
            case 4: f_step<4, DGRAD>(acc, as, bs, tx, ty); break;
            case 5: f_step<5, DGRAD>(acc, as, bs, tx, ty); break;
            case 6: f_step<6, DGRAD>(acc, as, bs, tx, ty); break;
            case 7: f_step<7, DGRAD>(acc, as, bs, tx, ty); break;
            default: f_step<8, DGRAD>(acc, as, bs, tx, ty); break;
        }
        if (++stage == F_STAGES) stage = 0;
        if (++it_c == chunks || st + 1 == steps) {
            // the block's sums go to their rows; the barrier of the next step lies between this and the next block's
            const int k = it >> 16, p0 = (it >> 8) & 255;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = ty + 8 * i;
                if (r < len) {
                    float* o = s_out + s_row[k * bm + p0 + r] * F_OSTR;
                    if constexpr (DGRAD) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            float lo, hi;
                            f2_unpack(acc.v[i][q], lo, hi);
                            o[tx + 16 * q] += lo + hi;
                        }
                    } else {
                        float4* o4 = reinterpret_cast<float4*>(o + tx * 4);
                        float4 v = *o4, u;
                        f2_unpack(acc.v[i][0], u.x, u.y);
                        f2_unpack(acc.v[i][1], u.z, u.w);
                        v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
                        *o4 = v;
                    }
                }
#pragma unroll
                for (int q = 0; q < (DGRAD ? 4 : 2); ++q) acc.v[i][q] = 0;
            }
            it_c = 0;
            ++it_i;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (G > 1) f_cluster_sync(); else __syncthreads();

    // ---- sums of the tile's CTAs, CTA 0 first, + bias; each CTA finishes its share of the tile
    const uint32_t local = f_smem(s_out);
    for (int e = grp * F_THREADS + tid; e < bm * (F_BN / 4); e += G * F_THREADS) {
        const int r = e / (F_BN / 4), c4 = (e % (F_BN / 4)) * 4;
        const long row = row0 + r;
        const int col = n0 + c4;
        if (row >= n || col >= cn) continue;
        float4 s;
        if (G == 1) {
            s = *reinterpret_cast<const float4*>(s_out + r * F_OSTR + c4);
        } else {
            s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int p = 0; p < G; ++p) {
                uint32_t peer;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(local + (r * F_OSTR + c4) * 4), "r"(p));
                float4 v;
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(peer) : "memory");
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
        }
        if (!DGRAD && bias != nullptr) {
            const float4 b4 = __ldg(reinterpret_cast<const float4*>(bias + col));
            s.x += b4.x; s.y += b4.y; s.z += b4.z; s.w += b4.w;
        }
        *reinterpret_cast<float4*>(out + row * cn + col) = s;
    }
    if (G > 1) f_cluster_sync();      // nobody leaves while a peer may still read its shared memory
}

// ---------------------------------------------------------------------------------------------------------
// weight gradient
// ---------------------------------------------------------------------------------------------------------
constexpr int FW_SEG = 512;               // tokens whose pairs are listed at a time

struct WgradSmem {
    float a[F_STAGES][F_BK * 64];         // x rows:  [pair][64 channels in]
    float b[F_STAGES][F_BK * 64];         // gy rows: [pair][64 channels out]
    int i[FW_SEG], j[FW_SEG];             // the segment's pairs, ascending
    int cnt[F_THREADS / 32];
};

// grid.x: (tap, 64 x 64 tile of its gradient), then - when the bias gradient is asked for - 64-column blocks of gy;
// grid.y: ranges of tokens.  Partials to ws_w[range][kk][cin][cout], ws_b[range][cout].
__global__ void __launch_bounds__(F_THREADS, 4)
wgrad_f32_kernel(const float* __restrict__ gy, const float* __restrict__ x, const int32_t* __restrict__ nbr,
                 float* __restrict__ ws_w, float* __restrict__ ws_b, long n, int cin, int cout, int kk, int tpb,
                 long rows_per_split, int tiles_m, int tiles_n) {
    extern __shared__ __align__(16) unsigned char f_smem_raw[];
    WgradSmem& sm = *reinterpret_cast<WgradSmem*>(f_smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = tid & 15, ty = tid >> 4;      // rows ty * 8 .. + 7, columns tx * 4 .. + 3
    const long i_begin = (long)blockIdx.y * rows_per_split, i_end = min(n, i_begin + rows_per_split);
    int tile = blockIdx.x;
    if (tile >= kk * tiles_m * tiles_n) {
        // column sums of gy: four columns and every eighth row per thread, the eight summed in order
        const int bx = tid & 15, by = tid >> 4, col = (tile - kk * tiles_m * tiles_n) * 64 + bx * 4;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (col < cout) {
#pragma unroll 8
            for (long i = i_begin + by; i < i_end; i += 8) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(gy + i * cout + col));
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
        }
        float4* part = reinterpret_cast<float4*>(sm.a[0]);
        part[tid] = s;
        __syncthreads();
        if (by == 0 && col < cout) {
            s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float4 v = part[q * 16 + bx];
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
            *reinterpret_cast<float4*>(ws_b + (long)blockIdx.y * cout + col) = s;
        }
        return;
    }
    const int tn = tile % tiles_n;
    tile /= tiles_n;
    const int tm = tile % tiles_m, k = tile / tiles_m;
    const int m0 = tm * 64, n0 = tn * 64;

    f2 acc[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[i][j] = 0;

    for (long seg = i_begin; seg < i_end; seg += FW_SEG) {
        // ---- the segment's pairs: a warp lists a quarter of it, then the quarters close up
        const long seg_end = min(i_end, seg + FW_SEG);
        int jj[FW_SEG / F_THREADS];
#pragma unroll
        for (int q = 0; q < FW_SEG / F_THREADS; ++q) {
            const long i = seg + warp * (FW_SEG / 4) + q * 32 + lane;
            jj[q] = i < seg_end ? __ldg(nbr + i * kk + k) : -1;
        }
        int cnt = 0;
#pragma unroll
        for (int q = 0; q < FW_SEG / F_THREADS; ++q) {
            const long i = seg + warp * (FW_SEG / 4) + q * 32 + lane;
            const long j = (long)jj[q] + (tpb > 0 ? (i / tpb) * (long)tpb : 0);
            const bool there = jj[q] >= 0 && j < n;
            jj[q] = there ? (int)j : -1;
            cnt += __popc(__ballot_sync(0xffffffffu, there));
        }
        if (lane == 0) sm.cnt[warp] = cnt;
        __syncthreads();
        int at = 0, pairs = 0;
#pragma unroll
        for (int q = 0; q < F_THREADS / 32; ++q) {
            at += q < warp ? sm.cnt[q] : 0;
            pairs += sm.cnt[q];
        }
#pragma unroll
        for (int q = 0; q < FW_SEG / F_THREADS; ++q) {
            const unsigned m = __ballot_sync(0xffffffffu, jj[q] >= 0);
            if (jj[q] >= 0) {
                const int p = at + __popc(m & ((1u << lane) - 1u));
                sm.i[p] = (int)(seg + warp * (FW_SEG / 4) + q * 32 + lane);
                sm.j[p] = jj[q];
            }
            at += __popc(m);
        }
        __syncthreads();
        const int steps = (pairs + F_BK - 1) / F_BK;
        auto load_stage = [&](int st) {
            const uint32_t a_base = f_smem(sm.a[st % F_STAGES]), b_base = f_smem(sm.b[st % F_STAGES]);
#pragma unroll
            for (int q = 0; q < F_BK * 16 / F_THREADS; ++q) {
                const int g = tid + q * F_THREADS;
                const int r = g >> 4, ch = (g & 15) * 4, p = st * F_BK + r;
                const bool in = p < pairs;
                const bool oka = in && m0 + ch < cin, okb = in && n0 + ch < cout;
                f_cp16(a_base + (r * 64 + ch) * 4, oka ? x + (long)sm.j[p] * cin + m0 + ch : x, oka ? 16u : 0u);
                f_cp16(b_base + (r * 64 + ch) * 4, okb ? gy + (long)sm.i[p] * cout + n0 + ch : gy, okb ? 16u : 0u);
            }
        };
#pragma unroll
        for (int s = 0; s < F_STAGES - 1; ++s) {
            if (s < steps) load_stage(s);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        for (int st = 0; st < steps; ++st) {
            asm volatile("cp.async.wait_group %0;" ::"n"(F_STAGES - 2) : "memory");
            __syncthreads();
            if (st + F_STAGES - 1 < steps) load_stage(st + F_STAGES - 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            const float* as = sm.a[st % F_STAGES] + ty * 8;
            const float* bs = sm.b[st % F_STAGES] + tx * 4;
#pragma unroll 8
            for (int p = 0; p < F_BK; ++p) {
                const float4 a0 = *reinterpret_cast<const float4*>(as + p * 64), a1 = *reinterpret_cast<const float4*>(as + p * 64 + 4);
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bs + p * 64);
                const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const f2 a = f2_pack(av[i], av[i]);
                    f2_fma(acc[i][0], a, b.x);
                    f2_fma(acc[i][1], a, b.y);
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();          // the lists and the ring are free for the next segment
    }
    float* dst = ws_w + ((long)blockIdx.y * kk + k) * cin * cout;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int ci = m0 + ty * 8 + i, co = n0 + tx * 4;
        float4 v;
        f2_unpack(acc[i][0], v.x, v.y);
        f2_unpack(acc[i][1], v.z, v.w);
        if (ci < cin && co < cout) *reinterpret_cast<float4*>(dst + (long)ci * cout + co) = v;
    }
}

// fixed-order sum of the ranges' partials, four elements per thread; the bias gradient behind the weights
__global__ void __launch_bounds__(128)
wgrad_f32_sum_kernel(const float* __restrict__ ws_w, const float* __restrict__ ws_b, int splits, float* __restrict__ gw,
                     float* __restrict__ gb, long n_w, int cout) {
    long e = (blockIdx.x * 128l + threadIdx.x) * 4;
    const float* src = ws_w;
    float* dst = gw;
    long stride = n_w;
    if (e >= n_w) {
        e -= n_w;
        if (gb == nullptr || e >= cout) return;
        src = ws_b; dst = gb; stride = cout;
    }
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int q = 0; q < splits; ++q) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(src + q * stride + e));
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    *reinterpret_cast<float4*>(dst + e) = s;
}

// ---------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------
// cudaFuncSetAttribute once per kernel and device (`ready`: the kernel's own set of devices)
static int f32_allow_smem(const void* kern, size_t bytes, std::atomic<uint64_t>& ready) {
    int dev = 0;
    SV_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if (ready.load() & bit) return SVTAD_OK;
    SV_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    ready.fetch_or(bit);
    return SVTAD_OK;
}

static size_t conv_f32_smem(int bm, int kk) {
    return sizeof(FwdRing) + (size_t)bm * F_OSTR * sizeof(float) + (size_t)kk * bm * 5;
}

template <bool DGRAD>
static int launch_conv_f32(const ConvArgs& p, const int32_t* status, int bm, int G, cudaStream_t s) {
    auto kern = conv_f32_kernel<DGRAD>;
    static std::atomic<uint64_t> ready{0};
    int rc = f32_allow_smem(reinterpret_cast<const void*>(kern), conv_f32_smem(128, F_MAX_KK), ready);
    if (rc) return rc;
    const int cn = DGRAD ? p.cin : p.cout, cred = DGRAD ? p.cout : p.cin;
    const int tiles_m = (int)((p.n + bm - 1) / bm), tiles_n = (cn + F_BN - 1) / F_BN;
    SV_CUDA(launch_plain(kern, dim3((unsigned)(tiles_m * tiles_n * G)), dim3(F_THREADS), conv_f32_smem(bm, p.kk), s, G,
                         (const float*)p.a, p.nbr, (const float*)p.w, (const float*)p.bias, (float*)p.out, status, (long)p.n, cred,
                         cn, p.cin, p.cout, p.kk, p.tpb, tiles_n, bm, G));
    return SVTAD_OK;
}

// Three CTAs fit an SM (444 in all).  Tiles of 128 rows waste least on the ends of the lists and read the weights least
// often, but only where they fill the GPU; otherwise 64 rows.  The steps of a tile are split over as many CTAs as bring
// the grid to about three CTAs an SM (clusters of up to three), or to two with larger clusters, which are harder to
// place: a full load of clusters of six took 22 us where 16 us were measured at two CTAs an SM.
template <bool DGRAD>
static int dispatch_conv_f32(const ConvArgs& p, const int32_t* status, cudaStream_t s) {
    const long tiles_n = ((DGRAD ? p.cin : p.cout) + F_BN - 1) / F_BN;
    const long t128 = (p.n + 127) / 128 * tiles_n, t64 = (p.n + 63) / 64 * tiles_n;
    const long sms = tc_num_sms();
    const int bm = t128 >= sms ? 128 : 64;
    const long tiles = bm == 128 ? t128 : t64;
    const long three = (3 * sms + tiles / 2) / tiles, two = (2 * sms + tiles / 2) / tiles;
    long G = three < 3 ? three : 3;
    if (two > G) G = two < 8 ? two : 8;
    return launch_conv_f32<DGRAD>(p, status, bm, G < 1 ? 1 : (int)G, s);
}

bool f32_supported(int cin, int cout, int kk, int dtype) {
    return dtype == SVTAD_F32 && cin % 4 == 0 && cout % 4 == 0 && kk <= F_MAX_KK;
}

static bool use_f32_tc(int op, int64_t n, int cin, int cout, int kk) { return forced_path() != 1 && f32_tc_wanted(op, n, cin, cout, kk); }

int f32_fwd(const ConvArgs& p, cudaStream_t s) {
    return use_f32_tc(SVTAD_OP_FWD, p.n, p.cin, p.cout, p.kk) ? f32_tc_fwd(p, s) : dispatch_conv_f32<false>(p, nullptr, s);
}
int f32_dgrad(const ConvArgs& p, const int32_t* status, cudaStream_t s) {
    return use_f32_tc(SVTAD_OP_DGRAD, p.n, p.cin, p.cout, p.kk) ? f32_tc_dgrad(p, status, s) : dispatch_conv_f32<true>(p, status, s);
}

// Token ranges: about two full loads of the GPU (four CTAs an SM), so that the centre tap's CTAs, which have every token
// for a pair, do not outlast the rest; each range at least 128 tokens, the partials of several ranges at most 31 MB, which
// with the bias gradient's fit the built-in workspace of svtad_conv_wgrad_static.
static int f32_wgrad_splits(int64_t n, int cin, int cout, int kk) {
    const long tiles = (long)kk * ((cin + 63) / 64) * ((cout + 63) / 64);
    const long by_rows = (n + 127) / 128, by_size = (31l << 20) / ((long)kk * cin * cout * 4);
    long s = (8l * tc_num_sms() + tiles - 1) / tiles;
    if (s > by_rows) s = by_rows;
    if (s > by_size) s = by_size;
    return (int)(s < 1 ? 1 : s);
}

size_t f32_wgrad_ws_bytes(int64_t n, int cin, int cout, int kk) {
    const size_t s = (size_t)f32_wgrad_splits(n, cin, cout, kk);
    return align_up(s * kk * cin * cout * sizeof(float), 256) + align_up(s * cout * sizeof(float), 256);
}

int f32_wgrad(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n, int cin, int cout, int kk,
              int tpb, void* ws, size_t ws_bytes, cudaStream_t s) {
    const size_t need = f32_wgrad_ws_bytes(n, cin, cout, kk);
    if (ws_bytes < need)
        return set_error(SVTAD_ERR_WORKSPACE, "svtad_conv_wgrad: workspace %zu < %zu bytes", ws_bytes, need);
    const int splits = f32_wgrad_splits(n, cin, cout, kk);
    const long n_w = (long)kk * cin * cout, rows = (n + splits - 1) / splits;
    float* ws_w = static_cast<float*>(ws);
    float* ws_b = reinterpret_cast<float*>(static_cast<char*>(ws) + align_up((size_t)splits * n_w * sizeof(float), 256));
    if (use_f32_tc(SVTAD_OP_WGRAD, n, cin, cout, kk)) return f32_tc_wgrad(gy, x, nbr, gw, gb, n, cin, cout, kk, tpb, ws_w, ws_b, splits, s);
    static std::atomic<uint64_t> ready{0};
    int rc = f32_allow_smem(reinterpret_cast<const void*>(wgrad_f32_kernel), sizeof(WgradSmem), ready);
    if (rc) return rc;
    const int tiles_m = (cin + 63) / 64, tiles_n = (cout + 63) / 64;
    dim3 grid((unsigned)(kk * tiles_m * tiles_n + (gb ? tiles_n : 0)), (unsigned)splits);
    wgrad_f32_kernel<<<grid, F_THREADS, sizeof(WgradSmem), s>>>((const float*)gy, (const float*)x, nbr, ws_w, ws_b, (long)n,
                                                               cin, cout, kk, tpb, rows, tiles_m, tiles_n);
    SV_LAUNCH_CHECK("wgrad_f32_kernel");
    const long quads = (n_w + (gb ? cout : 0)) / 4;
    wgrad_f32_sum_kernel<<<(unsigned)((quads + 127) / 128), 128, 0, s>>>(ws_w, ws_b, splits, (float*)gw, (float*)gb, n_w, cout);
    SV_LAUNCH_CHECK("wgrad_f32_sum_kernel");
    return SVTAD_OK;
}

// ---------------------------------------------------------------------------------------------------------
// FFMA rate of the device: what the CUDA-core kernels are measured against
// ---------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) ffma_peak_kernel(float* out, int iters, float seed) {
    float a[8], b = seed, c = 1.0f - seed * 0.5f;
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = seed + i;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = fmaf(a[i], b, c);     // 8 independent chains per thread
        }
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += a[i];
    if (s == 123.456f) out[0] = s;     // never true; keeps the loop alive
}

}  // namespace svtad

using namespace svtad;

// Launches `launches` timing kernels of iters * 64 FMAs per thread on ctas * 256 threads.  The caller times the
// launch (events on `stream`) and divides: flops = 2 * 64 * iters * ctas * 256 per launch.
extern "C" int svtad_ffma_probe(int ctas, int iters, float* scratch, void* stream) {
    SV_CHECK_ARG(ctas > 0 && iters > 0 && scratch != nullptr, "svtad_ffma_probe: bad arguments");
    ffma_peak_kernel<<<ctas, 256, 0, (cudaStream_t)stream>>>(scratch, iters, 0.999f);
    SV_LAUNCH_CHECK("ffma_peak_kernel");
    return SVTAD_OK;
}
