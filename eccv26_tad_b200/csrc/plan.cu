// Work plan of a neighbor table: what lets the large layers skip the neighbors that are not there.
//
// With tokens kept at random, 3.1 of 9 taps are there at keep 30 %, but a tile of 128 rows in their natural order has
// some row for every tap.  The plan
//   * orders the rows so that those with the same neighbors sit together: a counting sort by the eight bits of the ring
//     around the centre, in Gray-code order, so that neighbouring groups differ in one tap.  A tile then needs 3.8 taps
//     instead of 9 (18 880 rows, keep 30 %; 5.9 at keep 55 %) - and for the weight gradient
//   * lists per tap the (row, neighbor) pairs that exist.
// Any permutation is a correct order, and a row's own sum does not depend on it: taps that a tile skips would have added
// zeros.
//
// One launch of clusters of eight CTAs: one sorts, one per tap lists.  Latency bounds it (18 880 rows: a table of
// 680 KB); every row is looked at twice, the counts meet in distributed shared memory in between.
#include <atomic>

#include "plan.cuh"

namespace svtad {

constexpr int PLAN_THREADS = 1024, PLAN_G = 8, PLAN_WARPS = PLAN_THREADS / 32;

__device__ __forceinline__ uint32_t p_remote(const void* p, int cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(cta));
    return r;
}
__device__ __forceinline__ int p_load_remote(const int* p, int cta) {
    int v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(p_remote(p, cta)) : "memory");
    return v;
}
__device__ __forceinline__ void p_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct PlanRing { int tap[8]; int count; };      // the taps that make a row's key

struct PlanOut {
    int32_t* order; uint64_t* mask; int32_t* seq; int32_t* count; int32_t* pair_i; int32_t* pair_j;
};

struct SortSmem {
    uint16_t hist[PLAN_WARPS][256];     // per warp: rows per key, then the warp's next free place within the key
    int part[4][256];                   // rows per key and eight warps
    int total[256];                     // this CTA's rows per key
    int base[256];                      // first place of this CTA's rows of a key
    uint32_t taps[PLAN_MAX_ROWS / PLAN_TILE];
    uint8_t key[PLAN_MAX_ROWS / PLAN_G];
};

__device__ __forceinline__ int scan32(int v) {      // inclusive, over the warp
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += t;
    }
    return v;
}

// lanes of `among` that have this lane's key; eight ballots (__match_any_sync took 2 000 cycles where these take 300, with 32 warps
// on the SM and 20 different keys in a warp)
__device__ __forceinline__ unsigned same_key(int key, unsigned among) {
    unsigned same = among;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const unsigned set = __ballot_sync(0xffffffffu, key >> q & 1);
        same &= key >> q & 1 ? set : ~set;
    }
    return same;
}

__device__ void list_tap(const int32_t* __restrict__ nbr, long n, int kk, int tpb, int k, const PlanOut& o, int* s_w) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cta = blockIdx.x % PLAN_G;
    const long groups = (n + 31) / 32, per_warp = (groups + PLAN_G * PLAN_WARPS - 1) / (PLAN_G * PLAN_WARPS);
    const long g0 = (cta * PLAN_WARPS + warp) * per_warp, g1 = min(groups, g0 + per_warp);
    auto entry = [&](long g, int& j) {
        const long i = g * 32 + lane;
        const int raw = i < n ? __ldg(nbr + i * kk + k) : -1;
        const long jj = (long)raw + (tpb > 0 ? (i / tpb) * (long)tpb : 0);
        j = (int)jj;
        return raw >= 0 && jj < n;
    };
    int cnt = 0, j;
#pragma unroll 4
    for (long g = g0; g < g1; ++g) cnt += __popc(__ballot_sync(0xffffffffu, entry(g, j)));
    if (lane == 0) s_w[warp] = cnt;
    __syncthreads();
    const int incl = scan32(s_w[lane]);                         // 32 warps
    const int all = __shfl_sync(0xffffffffu, incl, 31);
    int at = __shfl_sync(0xffffffffu, incl, warp) - cnt;
    if (threadIdx.x == 0) s_w[PLAN_WARPS] = all;
    p_cluster_sync();
    const int theirs = lane < PLAN_G ? p_load_remote(&s_w[PLAN_WARPS], lane) : 0;
    at += __reduce_add_sync(0xffffffffu, lane < cta ? theirs : 0);
    const int total = __reduce_add_sync(0xffffffffu, theirs);
    if (cta == 0 && threadIdx.x == 0) o.count[k] = total;
    int32_t* pi = o.pair_i + (long)k * n;
    int32_t* pj = o.pair_j + (long)k * n;
#pragma unroll 4
    for (long g = g0; g < g1; ++g) {
        const bool there = entry(g, j);
        const unsigned m = __ballot_sync(0xffffffffu, there);
        if (there) {
            const int p = at + __popc(m & ((1u << lane) - 1u));
            pi[p] = (int)(g * 32 + lane);
            pj[p] = j;
        }
        at += __popc(m);
    }
    p_cluster_sync();          // nobody leaves while a peer may still read its counts
}

__device__ void sort_rows(const int32_t* __restrict__ nbr, long n, int kk, const PlanRing& ring, const PlanOut& o, SortSmem& sm,
                          int* s_w) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cta = blockIdx.x % PLAN_G;
    const unsigned lt = (1u << lane) - 1u;
    const int tiles = (int)((n + PLAN_TILE - 1) / PLAN_TILE);
    const long groups = (n + 31) / 32, per_warp = (groups + PLAN_G * PLAN_WARPS - 1) / (PLAN_G * PLAN_WARPS);
    const long g0 = (cta * PLAN_WARPS + warp) * per_warp, g1 = min(groups, g0 + per_warp);
    uint8_t* my_key = sm.key + warp * per_warp * 32;
    for (int b = lane; b < 256; b += 32) sm.hist[warp][b] = 0;
    __syncwarp();
#pragma unroll 2
    for (long g = g0; g < g1; ++g) {
        const long i = g * 32 + lane;
        int key = 0;
        if (i < n) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q < ring.count && __ldg(nbr + i * kk + ring.tap[q]) >= 0) key |= 1 << q;
            // place of this pattern in the Gray code sequence
            key ^= key >> 1;
            key ^= key >> 2;
            key ^= key >> 4;
        }
        my_key[(g - g0) * 32 + lane] = (uint8_t)key;
        const unsigned same = same_key(key, __ballot_sync(0xffffffffu, i < n));
        if (i < n && (same & lt) == 0) sm.hist[warp][key] += (uint16_t)__popc(same);
        __syncwarp();
    }
    __syncthreads();
    {
        // per key the warps' first places: four threads take eight warps each
        const int key = tid & 255, w0 = (tid >> 8) * 8;
        int c[8], run = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            c[w] = sm.hist[w0 + w][key];
            run += c[w];
        }
        sm.part[tid >> 8][key] = run;
        __syncthreads();
        int at = 0, sum = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            at += q < (tid >> 8) ? sm.part[q][key] : 0;
            sum += sm.part[q][key];
        }
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            sm.hist[w0 + w][key] = (uint16_t)at;
            at += c[w];
        }
        if (tid < 256) sm.total[key] = sum;
    }
    p_cluster_sync();
    int all = 0, below = 0, start = 0;
    if (tid < 256) {
#pragma unroll
        for (int g = 0; g < PLAN_G; ++g) {
            const int c = p_load_remote(&sm.total[tid], g);
            all += c;
            below += g < cta ? c : 0;
        }
        start = scan32(all);
        if (lane == 31) s_w[warp] = start;
        start -= all;
    }
    __syncthreads();
    if (tid < 256) {
        for (int w = 0; w < warp; ++w) start += s_w[w];
        sm.base[tid] = start + below;
    }
    for (int t = tid; t < tiles; t += PLAN_THREADS) sm.taps[t] = 0;
    __syncthreads();
    for (long g = g0; g < g1; ++g) {
        const long i = g * 32 + lane;
        const int key = my_key[(g - g0) * 32 + lane];
        const unsigned same = same_key(key, __ballot_sync(0xffffffffu, i < n));
        const int free_at = sm.hist[warp][key];
        __syncwarp();
        if (i < n) {
            o.order[sm.base[key] + free_at + __popc(same & lt)] = (int)i;
            if ((same & lt) == 0) sm.hist[warp][key] = (uint16_t)(free_at + __popc(same));
        }
        __syncwarp();
    }
    if (cta == 0) {
        // which taps a tile needs, and the tiles by how many those are
        for (long r = n + tid; r < (long)tiles * PLAN_TILE; r += PLAN_THREADS) o.order[r] = -1;
        if (tid < 256 && all > 0) {
            const uint32_t bits = tid ^ (tid >> 1);
            for (int t = start / PLAN_TILE; t <= (start + all - 1) / PLAN_TILE; ++t) atomicOr(&sm.taps[t], bits);
        }
        __syncthreads();
        uint64_t always = kk >= 64 ? ~0ull : (1ull << kk) - 1;
        uint64_t bit[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            bit[q] = q < ring.count ? 1ull << ring.tap[q] : 0;
            always &= ~bit[q];
        }
        for (int t = tid; t < tiles; t += PLAN_THREADS) {
            uint64_t m = always;
            const uint32_t taps = sm.taps[t];
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (taps >> q & 1u) m |= bit[q];
            o.mask[t] = m != 0 ? m : 1;          // a tile's sums have to be begun by some tap
        }
        // a warp per number of taps counts its tiles, then writes them behind those with more
        int mine = 0;
        if (warp <= 8)
            for (int t0 = 0; t0 < tiles; t0 += 32)
                mine += __popc(__ballot_sync(0xffffffffu, t0 + lane < tiles && __popc(sm.taps[t0 + lane]) == 8 - warp));
        if (lane == 0) s_w[warp] = mine;
        __syncthreads();
        if (warp <= 8) {
            int at = __reduce_add_sync(0xffffffffu, lane < warp ? s_w[lane] : 0);
            for (int t0 = 0; t0 < tiles; t0 += 32) {
                const bool here = t0 + lane < tiles && __popc(sm.taps[t0 + lane]) == 8 - warp;
                const unsigned m = __ballot_sync(0xffffffffu, here);
                if (here) o.seq[at + __popc(m & lt)] = t0 + lane;
                at += __popc(m);
            }
        }
    }
    p_cluster_sync();
}

__global__ void __launch_bounds__(PLAN_THREADS)
plan_kernel(const int32_t* __restrict__ nbr, long n, int kk, int tpb, int sorts, PlanRing ring, PlanOut o) {
    extern __shared__ __align__(16) unsigned char p_smem[];
    __shared__ int s_w[PLAN_WARPS + 1];
    const int job = blockIdx.x / PLAN_G + (sorts ? 0 : 1);
    pdl_wait();
    pdl_trigger();
    if (job == 0) sort_rows(nbr, n, kk, ring, o, *reinterpret_cast<SortSmem*>(p_smem), s_w);      // the longest first
    else list_tap(nbr, n, kk, tpb, job - 1, o, s_w);
}

}  // namespace svtad

using namespace svtad;

extern "C" size_t svtad_plan_bytes(int64_t n, int kk) {
    return n > 0 && n <= PLAN_MAX_ROWS && kk > 0 && kk <= 49 ? plan_layout(n, kk, nullptr, nullptr) : 0;
}

extern "C" const int32_t* svtad_plan_counts(const void* plan, int64_t n, int kk) {
    PlanView v;
    plan_layout(n, kk, plan, &v);
    return v.count;
}

extern "C" int svtad_plan_build(const int32_t* nbr, int64_t n, int kk, int tokens_per_batch, void* plan, void* stream) {
    return svtad_plan_build_parts(nbr, n, kk, tokens_per_batch, SVTAD_PLAN_ROWS | SVTAD_PLAN_PAIRS, plan, stream);
}

extern "C" int svtad_plan_build_parts(const int32_t* nbr, int64_t n, int kk, int tokens_per_batch, int parts, void* plan,
                                      void* stream) {
    SV_CHECK_ARG(svtad_plan_bytes(n, kk) > 0, "svtad_plan_build: no plan for %lld rows and %d taps", (long long)n, kk);
    SV_CHECK_ARG(nbr != nullptr && plan != nullptr && tokens_per_batch >= 0, "svtad_plan_build: bad argument");
    SV_CHECK_ARG(parts > 0 && parts <= (SVTAD_PLAN_ROWS | SVTAD_PLAN_PAIRS), "svtad_plan_build: no such parts: %d", parts);
    SV_CHECK_ARG(reinterpret_cast<uintptr_t>(plan) % 256 == 0, "svtad_plan_build: plan is not 256-byte aligned");
    PlanView v;
    plan_layout(n, kk, plan, &v);
    PlanOut o{const_cast<int32_t*>(v.order), const_cast<uint64_t*>(v.mask), const_cast<int32_t*>(v.seq),
              const_cast<int32_t*>(v.count), const_cast<int32_t*>(v.pair_i), const_cast<int32_t*>(v.pair_j)};
    // the ring around the centre of a square odd stencil; of any other one the first eight taps
    PlanRing ring{};
    int K = 1;
    while (K * K < kk) ++K;
    if (K * K == kk && K % 2 == 1 && K >= 3) {
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx)
                if (dy != 0 || dx != 0) ring.tap[ring.count++] = (dy + K / 2) * K + dx + K / 2;
    } else {
        while (ring.count < kk && ring.count < 8) { ring.tap[ring.count] = ring.count; ++ring.count; }
    }
    static std::atomic<uint64_t> ready{0};
    int dev = 0;
    SV_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if (!(ready.load() & bit)) {
        SV_CUDA(cudaFuncSetAttribute(plan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortSmem)));
        ready.fetch_or(bit);
    }
    const int sorts = parts & SVTAD_PLAN_ROWS ? 1 : 0, lists = parts & SVTAD_PLAN_PAIRS ? kk : 0;
    SV_CUDA(launch_pdl(plan_kernel, dim3((unsigned)((sorts + lists) * PLAN_G)), dim3(PLAN_THREADS), sorts ? sizeof(SortSmem) : 0,
                       (cudaStream_t)stream, PLAN_G, nbr, (long)n, kk, tokens_per_batch, sorts, ring, o));
    return SVTAD_OK;
}
