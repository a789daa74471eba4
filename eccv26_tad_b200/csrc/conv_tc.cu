// Host side of the tcgen05 / TMEM SparseConv2D path: the device error word, tensor-map encoding, tile
// and split planning, and the dispatch between the kernel families
//   conv_tc_hybrid.cu   one CTA per tile: gathered rows by per-warp cp.async, weight / gy tiles by TMA
//   conv_tc_pair.cu     forward / dgrad on CTA pairs (cta_group::2) where they are faster, see tc_choose()
// They replace opentad/models/bricks/implicit_gemm_v2.cu:197-417 (gather kernel + cuBLAS batched GEMM +
// reduce kernel) and the atomic backward kernels opentad/models/bricks/2d_sparse_v3.cu:656-745.
#include <cstdlib>
#include <cstring>
#include <atomic>
#include <map>
#include <mutex>
#include <utility>

#include "tc_common.cuh"

namespace svtad {

// Set (once, first code wins) by a bounded wait that gave up; read and cleared by svtad_device_error().
__device__ int g_tc_error = 0;

int* tc_error_ptr() {
    static thread_local int cached_dev = -1;
    static thread_local int* cached = nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    if (dev != cached_dev) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_tc_error) != cudaSuccess) return nullptr;
        cached = static_cast<int*>(p);
        cached_dev = dev;
    }
    return cached;
}

int tc_read_error(int32_t* code_out) {
    int v = 0;
    SV_CUDA(cudaDeviceSynchronize());
    SV_CUDA(cudaMemcpyFromSymbol(&v, g_tc_error, sizeof(int)));
    if (v != 0) {
        int zero = 0;
        SV_CUDA(cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(int)));
    }
    *code_out = v;
    return SVTAD_OK;
}

// SM count of the current device (cached per device ordinal; a racing first call stores the same value)
int tc_num_sms() {
    constexpr int MAX_DEV = 64;
    static int cached[MAX_DEV] = {0};
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (dev >= 0 && dev < MAX_DEV && cached[dev] > 0) return cached[dev];
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    if (dev >= 0 && dev < MAX_DEV) cached[dev] = v;
    return v;
}

// How many kernels the caller expects to share the GPU (svtad_set_concurrency; SVTAD_CONCURRENCY for a start value).
// The planning below then counts on SMs / share multiprocessors per kernel: fewer, longer CTAs (wide column blocks,
// several row tiles per persistent CTA, fewer token splits), which costs a kernel latency when it runs alone but
// saves SM time - every CTA pays about 7 us of set-up, first-operand latency and epilogue whatever its share of the
// work - when the SMs are contended anyway.
static std::atomic<int>& tc_share_ref() {
    static std::atomic<int> v{[] {
        const char* e = getenv("SVTAD_CONCURRENCY");
        int x = (e != nullptr && *e) ? atoi(e) : 1;
        return x < 1 ? 1 : (x > 16 ? 16 : x);
    }()};
    return v;
}
int tc_set_share(int n) {
    if (n < 1) n = 1;
    if (n > 16) n = 16;
    return tc_share_ref().exchange(n);
}
int tc_get_share() { return tc_share_ref().load(); }
// a lower bound on the share for the calling thread's next launches (svtad_conv_bwd runs its two kernels side by
// side and plans each for half the GPU even when the caller gave no hint)
static thread_local int t_share_floor = 1;
int tc_set_share_floor(int n) {
    const int old = t_share_floor;
    t_share_floor = n < 1 ? 1 : n;
    return old;
}
int tc_plan_sms() {
    const int g = tc_share_ref().load();
    int v = tc_num_sms() / (g > t_share_floor ? g : t_share_floor);
    return v < 8 ? 8 : v;
}

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) once per (kernel, device) instead of before every launch;
// the value only ever grows
int tc_ensure_smem(const void* kern, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, size_t> done;
    int dev = 0;
    SV_CUDA(cudaGetDevice(&dev));
    // what this thread has asked for lately needs no lock
    struct Seen { const void* kern; int dev; size_t bytes; };
    static thread_local Seen seen[64];
    Seen& hit = seen[(reinterpret_cast<uintptr_t>(kern) >> 4) % 64];
    if (hit.kern == kern && hit.dev == dev && hit.bytes >= bytes) return SVTAD_OK;
    std::lock_guard<std::mutex> hold(mu);
    auto key = std::make_pair(kern, dev);
    auto it = done.find(key);
    if (it == done.end() || it->second < bytes) {
        SV_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
        it = done.insert_or_assign(key, bytes).first;
    }
    hit = Seen{kern, dev, it->second};
    return SVTAD_OK;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

int tc_make_map(CUtensorMap* map, int rank, const void* base, const uint64_t* dims, const uint32_t* box, int fp16) {
    return tc_make_map_sw(map, rank, base, dims, box, fp16, 128);
}

int tc_make_map_sw(CUtensorMap* map, int rank, const void* base, const uint64_t* dims, const uint32_t* box, int type,
                   int swizzle_bytes) {
    // A descriptor depends only on (base, dims, box, element type, swizzle): a training step encodes the same few
    // again and again, so the last ones are kept per thread, found by a hash of these.
    struct Key { const void* base; uint64_t dims[3]; uint32_t box[3]; int rank, type, swz, dev; };
    struct Slot { Key key; CUtensorMap map; bool used; };
    constexpr unsigned SLOTS = 128;
    static thread_local Slot cache[SLOTS];
    Key key;
    memset(&key, 0, sizeof(key));
    key.base = base; key.rank = rank; key.type = type; key.swz = swizzle_bytes;
    uint64_t h = reinterpret_cast<uintptr_t>(base) >> 4;
    for (int i = 0; i < rank; ++i) {
        key.dims[i] = dims[i];
        key.box[i] = box[i];
        h = h * 0x9E3779B97F4A7C15ull + dims[i] * 8 + box[i];
    }
    if (cudaGetDevice(&key.dev) != cudaSuccess) key.dev = -1;
    Slot& slot = cache[(h ^ (h >> 29) ^ (h >> 47)) % SLOTS];
    if (slot.used && memcmp(&slot.key, &key, sizeof(Key)) == 0) { *map = slot.map; return SVTAD_OK; }
    EncodeTiledFn fn = encode_fn();
    if (fn == nullptr) return set_error(SVTAD_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    // the driver call needs this thread to hold the device's context (autograd worker threads may not yet)
    static thread_local int ctx_dev = -1;
    int dev = 0;
    SV_CUDA(cudaGetDevice(&dev));
    if (ctx_dev != dev) {
        SV_CUDA(cudaSetDevice(dev));   // binds the device's primary context to this thread; allocates nothing
        ctx_dev = dev;
    }
    cuuint64_t gdim[3], gstride[2];
    cuuint32_t bx[3], es[3] = {1, 1, 1};
    uint64_t stride = type == TC_MAP_F32 ? 4 : 2;
    for (int i = 0; i < rank; ++i) {
        gdim[i] = dims[i];
        bx[i] = box[i];
        stride *= dims[i];
        if (i < rank - 1) gstride[i] = stride;
    }
    CUresult r = fn(map, type == TC_MAP_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : type == 1 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank,
                    const_cast<void*>(base), gdim, gstride, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(SVTAD_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
    slot.key = key; slot.map = *map; slot.used = true;
    return SVTAD_OK;
}

// One CTA runs per SM, so the cost of a column-block width is
// (waves over the SMs) x (bytes a CTA stages per K step: 16 KB of gathered rows + its weight tile).
int tc_pick_bn(int cn, long m_tiles) {
    const int cand[5] = {256, 192, 128, 96, 64};
    const char* e = getenv("SVTAD_TC_BN");
    if (e != nullptr && *e) {
        int v = atoi(e);
        for (int c : cand)
            if (v == c && cn % v == 0) return v;
    }
    const long sms = tc_plan_sms();
    int best = 0;
    long best_cost = 0;
    for (int c : cand) {
        if (c - 64 >= cn) continue;          // no wider than the output rounded up to 64 columns
        long ctas = m_tiles * ((cn + c - 1) / c);
        long waves = (ctas + sms - 1) / sms;
        long cost = waves * (A_TILE_BYTES + b_tile_bytes_for(c));
        if (best == 0 || cost < best_cost) { best = c; best_cost = cost; }
    }
    return best;
}

// The column block that covers the output width in the least time, blocks times what a K step takes at that width, for kernels whose
// tiles fill the GPU whatever the width.  By least padding a width of 320 went in five blocks of 64, which gather a row tile five
// times: 37 760 rows, C = 320: forward 108 us, in two blocks of 192 68, a training pass 200 and 154; 34 560 rows, C = 448: 184 and 98.
int tc_widest_bn(int cn) {
    const int cand[4] = {256, 192, 128, 64};
    const char* e = getenv("SVTAD_TC_BN");
    if (e != nullptr && *e) {
        int v = atoi(e);
        for (int c : cand)
            if (v == c && cn % v == 0) return v;
    }
    const double step_us[4] = {0.344, 0.28, 0.23, 0.19};
    int best = 0;
    double least = 0;
    for (int i = 0; i < 4; ++i) {
        const double t = (cn + cand[i] - 1) / cand[i] * step_us[i];
        if (best == 0 || t < least) { best = cand[i]; least = t; }
    }
    return best;
}

// wgrad work split: (pairs of 64-channel blocks) x (column blocks of width BN) x (splits over tokens).
// A bias gradient takes one more half pair: a block of ones, whose rows of D are the column sums of gy - the spare half
// of the last pair where the block count is odd, else a pair of its own.  (At C = 1024 that pair costs 1.4 % of the
// kernel; a separate pass over gy plus the reduction of its partials took 86 + 30 us beside a 305 us main kernel.)
// One CTA runs per SM, so a candidate (BN, splits) costs
//   (waves over the SMs) x (64-token steps per CTA + fixed cost) x (cycles per step at that BN)
// plus the trip of the fp32 partials through memory (written by the main kernel, read by the reduction).
// Cycles per step and the partials' rate are what these kernels were measured at on a B200.
// limit: most bytes the partials of several splits may take (0: any).
static WgradPlan wgrad_plan_for(int64_t n, int cin, int cout, int kk, bool with_bias, long sms, size_t limit = 0) {
    const int nblocks = kk * ((cin + 63) / 64);
    long max_by_rows = (n + 2 * STAGE_K - 1) / (2 * STAGE_K);
    if (max_by_rows < 1) max_by_rows = 1;
    if (max_by_rows > 64) max_by_rows = 64;
    int forced_bn = 0;
    if (const char* e = getenv("SVTAD_TC_WGRAD_BN")) forced_bn = atoi(e);
    long forced_s = 0;
    if (const char* e = getenv("SVTAD_TC_WGRAD_SPLITS")) forced_s = atol(e);
    const int cand[4] = {256, 192, 128, 64};
    const double step_cycles[4] = {650.0, 584.0, 450.0, 400.0};
    // partials are written once and read once: from L2 while they fit beside the operands, else from memory
    const double partial_cycles_l2 = 2.0 * 1.9e9 / 12.0e12, partial_cycles_mem = 2.0 * 1.9e9 / 4.0e12;
    const double second_launch = 3000.0;
    WgradPlan best;
    best.bn = 0;
    double best_cost = 0;
    for (int ci = 0; ci < 4; ++ci) {
        const int bn = cand[ci];
        if (bn - 64 >= cout) continue;                                   // no wider than cout rounded up to 64 columns
        if (bn < 192 && best.bn != 0 && forced_bn == 0) continue;      // narrow blocks only when a wide one would be mostly padding
        if (forced_bn > 0 && bn != forced_bn && cout % forced_bn == 0) continue;
        WgradPlan pl;
        pl.bn = bn;
        pl.n_nblk = (cout + bn - 1) / bn;
        pl.n_pairs = with_bias ? nblocks / 2 + 1 : (nblocks + 1) / 2;
        pl.ones_block = with_bias;
        const long ctas = (long)pl.n_pairs * pl.n_nblk;
        for (long c = 1; c <= max_by_rows; ++c) {
            if (forced_s > 0 && c != (forced_s < max_by_rows ? forced_s : max_by_rows)) continue;
            const long tps = ((n + c - 1) / c + STAGE_K - 1) / STAGE_K * STAGE_K;
            const long splits = (n + tps - 1) / tps;
            if (limit > 0 && splits > 1 && tc_wgrad_partials(splits, with_bias, cin, cout, kk) > limit) continue;
            const long waves = (ctas * splits + sms - 1) / sms;
            const double steps = (double)tps / STAGE_K + 12.0;          // + set-up, first operands, drain
            // one split needs no partials and no second launch
            const double partial_bytes = splits > 1 ? (double)splits * kk * cin * cout * sizeof(float) : 0.0;
            const double cost = (double)waves * steps * step_cycles[ci] + (splits > 1 ? second_launch : 0.0) +
                                partial_bytes * (partial_bytes < 48e6 ? partial_cycles_l2 : partial_cycles_mem);
            if (best.bn == 0 || cost < best_cost * 0.98) {
                best = pl;
                best.tokens_per_split = tps;
                best.splits = (int)splits;
                best_cost = cost;
            }
        }
    }
    return best;
}

// The search above costs the host 1-20 us; the last few answers are kept per thread (a training step asks for the same
// few problems again and again).  Key 0 stands for the workspace size that covers every hint.
struct PlanMemo {
    int64_t n = -1;
    int cin, cout, kk;
    long key;
    WgradPlan plan;
    size_t bytes;
    bool is(int64_t n_, int cin_, int cout_, int kk_, long key_) const {
        return n == n_ && cin == cin_ && cout == cout_ && kk == kk_ && key == key_;
    }
};
static PlanMemo& plan_slot(int64_t n, int cin, int cout, int kk, long key) {
    constexpr unsigned SLOTS = 64;
    static thread_local PlanMemo memo[SLOTS];
    const uint64_t h = ((uint64_t)n * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)cin << 40) ^ ((uint64_t)cout << 20) ^ (uint64_t)(kk * 1024 + key);
    return memo[(h ^ (h >> 29) ^ (h >> 47)) % SLOTS];
}
static bool plan_overridden() { return getenv("SVTAD_TC_WGRAD_BN") != nullptr || getenv("SVTAD_TC_WGRAD_SPLITS") != nullptr; }

WgradPlan tc_wgrad_plan(int64_t n, int cin, int cout, int kk, bool with_bias, size_t limit) {
    const long sms = tc_plan_sms(), key = 2 * sms + with_bias;
    if (limit > 0) {
        const WgradPlan pl = tc_wgrad_plan(n, cin, cout, kk, with_bias, 0);
        return tc_wgrad_plan_bytes(pl, cin, cout, kk) <= limit ? pl : wgrad_plan_for(n, cin, cout, kk, with_bias, sms, limit);
    }
    if (plan_overridden()) return wgrad_plan_for(n, cin, cout, kk, with_bias, sms);
    PlanMemo& m = plan_slot(n, cin, cout, kk, key);
    if (!m.is(n, cin, cout, kk, key)) m = PlanMemo{n, cin, cout, kk, key, wgrad_plan_for(n, cin, cout, kk, with_bias, sms), 0};
    return m.plan;
}

size_t tc_wgrad_partials(long splits, bool with_bias, int cin, int cout, int kk) {
    return align_up((size_t)splits * kk * cin * cout * sizeof(float), 256) +
           (with_bias ? align_up((size_t)splits * cout * sizeof(float), 256) : 0);
}
size_t tc_wgrad_plan_bytes(const WgradPlan& pl, int cin, int cout, int kk) {
    return tc_wgrad_partials(pl.splits, pl.ones_block != 0, cin, cout, kk);
}

// What callers are told to provide: enough for the plan under every concurrency hint, so that a workspace
// sized once stays valid when the hint changes (a leaner plan usually has fewer token splits, but the waves'
// rounding can go the other way: 18 880 rows at C=192, 5x5 takes 3 splits planned for 148 SMs and 5 for 74).
size_t tc_wgrad_ws_bytes(int64_t n, int cin, int cout, int kk) {
    PlanMemo& m = plan_slot(n, cin, cout, kk, 0);
    if (!plan_overridden() && m.is(n, cin, cout, kk, 0)) return m.bytes;
    size_t need = 0;
    const int sms = tc_num_sms();
    for (int share = 1; share <= 16; ++share)
        for (int with_bias = 0; with_bias < 2; ++with_bias) {
            int v = sms / share;
            if (v < 8) v = 8;
            const size_t b = tc_wgrad_plan_bytes(wgrad_plan_for(n, cin, cout, kk, with_bias != 0, v), cin, cout, kk);
            if (b > need) need = b;
        }
    if (!plan_overridden()) m = PlanMemo{n, cin, cout, kk, 0, WgradPlan{}, need};
    return need;
}

// fixed-order reduction of the per-split partials (4 elements per thread), one rounding; OUT32: the rounded values are
// written as fp32 (the gradient of an fp32 master parameter), which saves a pass over the gradient
template <bool OUT32>
__global__ void __launch_bounds__(256)
wgrad_reduce4_kernel(const float* __restrict__ ws_w, int splits, const float* __restrict__ ws_b, int splits_b,
                     void* __restrict__ gw, void* __restrict__ gb, long n_w, int cout, int fp16) {
    pdl_wait();
    pdl_trigger();
    long e = (blockIdx.x * (long)blockDim.x + threadIdx.x) * 4;
    const float* src;
    void* base;
    long at;
    long stride;
    int cnt;
    if (e < n_w) {
        src = ws_w + e; base = gw; at = e; stride = n_w; cnt = splits;
    } else if (gb != nullptr && e - n_w < cout) {
        src = ws_b + (e - n_w); base = gb; at = e - n_w; stride = cout; cnt = splits_b;
    } else {
        return;
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int s = 0; s < cnt; ++s) {
        float4 v = __ldcg(reinterpret_cast<const float4*>(src + (long)s * stride));
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    uint2 o;
    o.x = pack2(acc.x, acc.y, fp16 != 0);
    o.y = pack2(acc.z, acc.w, fp16 != 0);
    if (OUT32) {
        auto wide = [&](uint32_t v) { return widen(static_cast<uint16_t>(v & 0xffffu), fp16 != 0); };
        *reinterpret_cast<float4*>(static_cast<float*>(base) + at) = make_float4(wide(o.x), wide(o.x >> 16), wide(o.y), wide(o.y >> 16));
    } else {
        *reinterpret_cast<uint2*>(static_cast<uint16_t*>(base) + at) = o;
    }
}


int tc_wgrad_reduce_launch(const float* ws_w, int splits, const float* ws_b, int splits_b, void* gw, void* gb,
                           long n_w, int cout, int fp16, bool out32, cudaStream_t s) {
    long total4 = (n_w + (gb ? cout : 0) + 3) / 4;
    SV_CUDA(launch_pdl(out32 ? wgrad_reduce4_kernel<true> : wgrad_reduce4_kernel<false>,
                      dim3((unsigned)((total4 + 255) / 256)), dim3(256), 0, s, 1, ws_w, splits, ws_b, splits_b, gw, gb, n_w,
                      cout, fp16));
    return SVTAD_OK;
}

bool tc_supported(int op, int64_t n, int cin, int cout, int kk, int dtype) {
    if (dtype != SVTAD_BF16 && dtype != SVTAD_F16) return false;
    if (n <= 0 || kk > 49) return false;
    // 32: the epilogue's column chunk; a row of 32 channels is 64 bytes, so rows stay 16-byte aligned for the copies
    if (cin % 32 != 0 || cout % 32 != 0) return false;
    (void)op;
    return true;
}

// Forward / dgrad on CTA pairs (tcgen05 cta_group::2) or on single CTAs.  A pair stages half of the weight tile per CTA, so
// its K steps are shorter; it starts later, and single CTAs may take narrower column blocks to fill the machine.  Times as
// measured on a B200 (us; rows, layer: pair, single): 18 880, 256 -> 256, 5x5: 40.9, 43.2; 14 160, 384, 5x5: 94.5, 108;
// 9 440, 384, 5x5: 50.4, 55.9; 18 880, 192, 3x3: 15.5, 14.5; 9 440, 768, 3x3: 79.1, 74.7; 37 760, 128, 3x3: 17.4, 16.8; 23 600,
// 256, 5x5: 74.1, 81.7; 37 760, 64, 5x5: 18.7, 18.0; 20 480, 1024 -> 32, 5x5: 163, 174; 9 984, 512, 7x7: 358, 266.  The two
// estimates below choose within 0.2 % of the faster one on average over 326 such calls (3x3 and 5x5); where they are close the
// kernel stays that was there first (pairs from as many row tiles as SMs on).  A tile whose K steps a cluster shares goes to
// single CTAs, and under a concurrency hint only the number of tiles counts.
// A row's sum is the same either way.  SVTAD_TC_IMPL=pair / hybrid overrides the choice.
static TcChoice choose(int64_t n, int cred, int cn, int kk, bool dgrad) {
    const long m_tiles = (n + TILE_M - 1) / TILE_M, sms = tc_num_sms();
    const int steps = kk * ((cred + STAGE_K - 1) / STAGE_K);
    TcChoice c{m_tiles > sms, 0, 1, 0.0};
    c.bn = hybrid_split(cn, m_tiles, steps, dgrad, c.split);
    if (c.bn != 0) c.pair = false;
    else c.bn = tc_pick_bn(cn, m_tiles);
    const char* e = getenv("SVTAD_TC_IMPL");
    const bool forced = e != nullptr && *e;
    if (forced) c.pair = e[0] == 'p';
    if (c.split == 1) {
        auto at = [](int bn) { return bn == 256 ? 4 : bn == 192 ? 3 : bn == 128 ? 2 : bn == 96 ? 1 : 0; };
        const double pair_step[5] = {0.20, 0.2375, 0.2375, 0.29, 0.316}, single_step[5] = {0.21, 0.245, 0.266, 0.352, 0.366};
        auto time = [&](double start, long items, long slots, double step) {
            const long waves = (items + slots - 1) / slots;
            return start + (double)waves * steps * step + (double)(waves - 1) * 1.7;
        };
        const int wide = tc_widest_bn(cn);
        // the tables of stencils beyond 5x5 leave pairs with 256 columns room for two rounds of buffers instead of three: 0.455 us a step
        const size_t table = 2 * (size_t)TILE_M * kk * sizeof(int) + 2048 + 512, stage = A_TILE_BYTES + (size_t)wide / 2 * 128;
        const double ring = (TC_SMEM_LIMIT - 1024 - table) / stage < 6 ? 1.44 : 1.0;
        const double pair = time(7.0, (m_tiles + 1) / 2 * ((cn + wide - 1) / wide), sms / 2, pair_step[at(wide)] * ring);
        const double single = time(5.2, m_tiles * ((cn + c.bn - 1) / c.bn), sms, single_step[at(c.bn)]);
        if (!forced && tc_plan_sms() == sms) c.pair = c.pair ? single >= 0.97 * pair : pair < 0.926 * single;
        c.us = pair < single ? pair : single;
    }
    return c;
}

// The estimates cost the host 0.4 us; the last few answers are kept per thread, as those of tc_wgrad_plan().
TcChoice tc_choose(int64_t n, int cred, int cn, int kk, bool dgrad) {
    if (getenv("SVTAD_TC_IMPL") != nullptr || getenv("SVTAD_TC_BN") != nullptr) return choose(n, cred, cn, kk, dgrad);
    struct Memo {
        int64_t n = -1;
        int cred, cn, kk, sms, all, dgrad;
        TcChoice choice;
    };
    constexpr unsigned SLOTS = 64;
    static thread_local Memo memo[SLOTS];
    const int sms = tc_plan_sms(), all = tc_num_sms();
    const uint64_t h = ((uint64_t)n * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)cred << 40) ^ ((uint64_t)cn << 20) ^ (uint64_t)(kk * 2048 + sms * 2 + dgrad);
    Memo& m = memo[(h ^ (h >> 29) ^ (h >> 47)) % SLOTS];
    if (m.n != n || m.cred != cred || m.cn != cn || m.kk != kk || m.sms != sms || m.all != all || m.dgrad != dgrad)
        m = Memo{n, cred, cn, kk, sms, all, dgrad, choose(n, cred, cn, kk, dgrad)};
    return m.choice;
}

int tc_fwd(const ConvArgs& p, cudaStream_t s) {
    if (p.plan == nullptr && tc_choose(p.n, p.cin, p.cout, p.kk, false).pair) return pair_fwd(p, s);
    return hybrid_fwd(p, s);
}

int tc_dgrad(const ConvArgs& p, const int32_t* status, cudaStream_t s) {
    if (p.plan == nullptr && tc_choose(p.n, p.cout, p.cin, p.kk, true).pair) return pair_dgrad(p, status, s);
    return hybrid_dgrad(p, status, s);
}

int tc_wgrad(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n, int cin, int cout,
             int kk, int tpb, int dtype, int grad_dtype, void* ws, size_t ws_bytes, bool fit, cudaStream_t s) {
    return hybrid_wgrad(gy, x, nbr, gw, gb, n, cin, cout, kk, tpb, dtype, grad_dtype, ws, ws_bytes, fit, s);
}

}  // namespace svtad
