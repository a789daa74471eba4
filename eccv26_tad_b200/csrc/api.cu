// C ABI of the SparseConv2D ops: argument validation, path selection, workspace layout.
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "tc_common.cuh"

namespace svtad {

static thread_local char g_err[512] = "";

int set_error(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

// 0 = automatic, 1 = force CUDA-core kernels, 2 = force tensor-core kernels
int forced_path() {
    const char* e = getenv("SVTAD_FORCE_PATH");
    if (e == nullptr || *e == 0) return 0;
    if (strcmp(e, "simt") == 0 || strcmp(e, "fp32") == 0) return 1;
    if (strcmp(e, "tc") == 0) return 2;
    return 0;
}

static bool use_tc(int op, int64_t n, int cin, int cout, int kk, int dtype) {
    int f = forced_path();
    if (f == 1) return false;
    return tc_supported(op, n, cin, cout, kk, dtype);
}

static int check_common(const char* who, int64_t n, int cin, int cout, int kk, int tpb, int dtype) {
    SV_CHECK_ARG(n >= 0 && n < (1ll << 31), "%s: n=%lld outside [0, 2^31)", who, (long long)n);
    SV_CHECK_ARG(cin > 0 && cout > 0, "%s: bad channel counts %d -> %d", who, cin, cout);
    SV_CHECK_ARG(kk > 0 && kk <= 49, "%s: kk=%d outside [1, 49]", who, kk);
    SV_CHECK_ARG(tpb >= 0, "%s: tokens_per_batch=%d is negative", who, tpb);
    SV_CHECK_ARG(dtype == SVTAD_F32 || dtype == SVTAD_BF16 || dtype == SVTAD_F16, "%s: unknown dtype %d", who, dtype);
    // same requirement as the reference wrapper (sparse_conv_layer.py:39-42)
    if (cin % 4 != 0)
        return set_error(SVTAD_ERR_UNSUPPORTED, "%s: C_in (%d) must be divisible by 4", who, cin);
    return SVTAD_OK;
}

static bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// Per device: a stream of the library's own and two events, used to run the weight gradient next to the
// input gradient inside svtad_conv_bwd.  Created on first use, never destroyed (process lifetime).
struct SideLane {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    std::mutex mu;     // one fork .. join sequence at a time per device (events are shared)
};
static constexpr int MAX_DEVICES = 64;
static SideLane g_lane[MAX_DEVICES];

static bool overlap_backward() {
    static const bool on = [] {
        const char* e = getenv("SVTAD_OVERLAP_BACKWARD");
        return !(e != nullptr && e[0] == '0');
    }();
    return on;
}

static int lane_ready(SideLane& l) {
    if (l.stream != nullptr) return SVTAD_OK;
    SV_CUDA(cudaStreamCreateWithFlags(&l.stream, cudaStreamNonBlocking));
    SV_CUDA(cudaEventCreateWithFlags(&l.fork, cudaEventDisableTiming));
    SV_CUDA(cudaEventCreateWithFlags(&l.join, cudaEventDisableTiming));
    return SVTAD_OK;
}

}  // namespace svtad

using namespace svtad;

extern "C" int svtad_version(void) { return 100; }

extern "C" const char* svtad_last_error_string(void) { return g_err; }

extern "C" int svtad_path_for(int op, int64_t n, int cin, int cout, int kk, int dtype) {
    return use_tc(op, n, cin, cout, kk, dtype) ? 1 : 0;
}

extern "C" int svtad_set_concurrency(int kernels) { return tc_set_share(kernels); }

extern "C" int svtad_get_concurrency(void) { return tc_get_share(); }

extern "C" int svtad_device_error(int32_t* code_out) {
    SV_CHECK_ARG(code_out != nullptr, "svtad_device_error: code_out is null");
    return tc_read_error(code_out);
}

// weight gradient alone, by a plan's pair lists or not
static size_t wgrad_ws_bytes(int64_t n, int cin, int cout, int kk, int dtype, bool by_pairs) {
    if (n <= 0 || cin <= 0 || cout <= 0 || kk <= 0) return 0;
    const bool tc = tc_supported(SVTAD_OP_WGRAD, n, cin, cout, kk, dtype);
    if (by_pairs && tc && forced_path() != 1 && pairs_wgrad_wanted(cin, kk)) return pairs_wgrad_ws_bytes(cin, cout);
    const size_t a = simt_wgrad_ws_bytes(n, cin, cout, kk, dtype), b = tc ? tc_wgrad_ws_bytes(n, cin, cout, kk) : 0;
    return a > b ? a : b;
}

extern "C" size_t svtad_workspace_bytes(int op, int64_t n, int cin, int cout, int kk, int dtype) {
    if (n <= 0 || cin <= 0 || cout <= 0 || kk <= 0) return 0;
    switch (op) {
        case SVTAD_OP_FWD: return 0;
        case SVTAD_OP_DGRAD: return align_up((size_t)n * cin * sizeof(float), 256);   // scatter form only
        case SVTAD_OP_WGRAD: return wgrad_ws_bytes(n, cin, cout, kk, dtype, false);
        case SVTAD_OP_BWD: {  // with or without a plan
            const size_t a = svtad_bwd_workspace_bytes(n, cin, cout, kk, dtype, 0, 1);
            const size_t b = svtad_bwd_workspace_bytes(n, cin, cout, kk, dtype, SVTAD_PLAN_PAIRS, 1);
            return a > b ? a : b;
        }
    }
    return 0;
}

extern "C" size_t svtad_bwd_workspace_bytes(int64_t n, int cin, int cout, int kk, int dtype, int plan_use, int scatter) {
    // both halves run at the same time: the two workspaces sit side by side
    return align_up(wgrad_ws_bytes(n, cin, cout, kk, dtype, (plan_use & SVTAD_PLAN_PAIRS) != 0), 256) +
           (scatter ? svtad_workspace_bytes(SVTAD_OP_DGRAD, n, cin, cout, kk, dtype) : 0);
}

// Which parts of a plan gain a layer more than it costs to make them for this one layer and call: the row order (forward,
// input gradient) takes 7 us at 4 720 rows, 12 at 18 880, 15 at 37 760, 24 at 75 520, and a few more for the kernel that
// starts cold behind it; the pair lists (weight gradient; 3 x 3) 4 to 15, next to the input gradient.  A tile of ordered rows
// needs about 1.2 times the taps that its rows have on average, so what the order saves goes by work * (1 - 1.2 density), and
// on what it costs the line rises with the rows.  Measured, us of a training pass (forward + backward, graph replays) without
// a plan and with one made for it, by that figure:
//   4 720 rows, C = 512, density 0.35 (13 GFLOP): 77 -> 80             11 800, C = 320, 0.35 (13): 90 -> 76
//   18 880, C = 256, 0.35 (13): 70 -> 85                              11 800, C = 384, 0.35 (18): 112 -> 82
//   75 520, C = 128, 0.35 (13): 95 -> 108                             4 720, C = 768, 0.35 (29): 152 -> 123
//   37 760, C = 192, 0.35 (15): 83 -> 81                              18 880, C = 384, 0.35 (29): 145 -> 106
//   21 600, C = 512, 0.55 (35): 258 -> 197                            37 760, C = 320, 0.35 (40): 218 -> 150
//   75 520, C = 192, 0.35 (29): 150 -> 139                            18 880, C = 1024, 0.35 (207): 768 -> 391
// With few tiles the longest one, which needs nearly every tap, is all that matters, and up to sixteen the kernels without a
// plan share a tile's K steps over a cluster: 1 770, C = 1024, 0.35 (19): 117 -> 140; 3 920, C = 1024, 0.51 (29): 183 -> 197.
// Stencils beyond 3 x 3: the order is by the eight nearest neighbors, and a tile needs nearly all of the others (19.9 of 25
// taps at density 0.28, 22.4 at 0.61): 2 360 rows, C = 512: forward 38 -> 78 us; 18 880, C = 256: 44 -> 43.  So these take the
// lists alone (8 to 30 us), which save work * (1 - density): 4 720 rows, C = 384, 0.28 (25 GFLOP): 138 -> 113; 9 440, C = 256, 0.28
// (22): 105 -> 111; 2 360, C = 512, 0.27 (22): 115 -> 131; 18 880, C = 256, 0.28 (45): 158 -> 148; 7 840, C = 512, 0.44 (58): 263 -> 226.
// density = pairs per row and tap; negative: not known, the sparse case (0.35) is assumed.
static double left_out(int64_t n, int cin, int cout, int kk, double there, double factor) {
    return 2e-9 * (double)n * kk * cin * cout * (1 - factor * there);
}
static double known_density(double density) { return density < 0 ? 0.35 : density < 1 ? density : 1; }

extern "C" int svtad_plan_wanted(int64_t n, int cin, int cout, int kk, int dtype, double density) {
    if (svtad_plan_bytes(n, kk) == 0 || kk < 2) return 0;
    const double there = known_density(density);
    const bool near = kk <= 9;
    const bool pays = near ? n > 2048 && (n > 4096 || there < 0.4) && left_out(n, cin, cout, kk, there, 1.2) >= 13.2 + (double)n / 5000
                           : left_out(n, cin, cout, kk, there, 1.0) >= 23 + (double)n / 2500;
    if (!pays || !use_tc(SVTAD_OP_FWD, n, cin, cout, kk, dtype)) return 0;
    return (near ? SVTAD_PLAN_ROWS : 0) | (pairs_wgrad_wanted(cin, kk) ? SVTAD_PLAN_PAIRS : 0);
}

// The same for a forward alone, which has to earn its row order by itself.  What the order saves is the share of the time that
// the kernel without one takes, which goes by its waves (8 736 rows, C = 384, are one wave of 70 tile pairs, 9 600 rows two).  us
// without and with an order made for the call, and in brackets what it is expected to save, before it is made:
//   12 960 rows, C = 512, density 0.55 (21): 56.5 -> 50.7        8 736, C = 384, 0.2 (18): 23.9 -> 28.7
//   11 800, C = 384, 0.35 (22): 34.8 -> 33.1                     18 880, C = 320, 0.35 (21): 36.0 -> 36.3
//   37 760, C = 320, 0.35 (40): 65.9 -> 53.1                     75 520, C = 256, 0.35 (36): 64.7 -> 67.0
// Where a CTA's share of the tiles is shorter than the longest tile, which needs every tap, that one decides: 18 940 rows, 512 ->
// 192, density 0.19: 30.9 -> 42.1; 8 960 rows, 640 -> 256, 0.19: 30.5 -> 37.7; 4 720, C = 768, 0.55: 43.4 -> 56.2.  There the
// order, 9 us and one per 3 200 rows, and that tile together have to be shorter than the kernel without.
// Of 1 129 forwards of 41 to 180 tiles, 256 to 1 024 -> 128 to 1 024 channels, that the first line takes, 123 lost 3 to 27 % (1.3 %
// from the better of the two on average), with the second 32 lose up to 17 % (0.4 %); of 926 up to 600 tiles 8 (0.07 %).
extern "C" int svtad_plan_wanted_fwd(int64_t n, int cin, int cout, int kk, int dtype, double density) {
    const int rows = svtad_plan_wanted(n, cin, cout, kk, dtype, density) & SVTAD_PLAN_ROWS;
    if (!rows || n <= 5120) return 0;
    const double there = known_density(density), without = tc_choose(n, cin, cout, kk, false).us;
    if (without * (1 - 1.1 * there) < 16 + (double)n / 3600) return 0;
    const double longest = hybrid_longest_us(n, cin, cout, kk, there);
    return longest == 0 || 9 + (double)n / 3200 + longest < 1.06 * without ? rows : 0;
}

extern "C" int svtad_conv_fwd(const void* x, const int32_t* nbr, const void* w, const void* bias,
                              void* y, int64_t n, int cin, int cout, int kk, int tokens_per_batch,
                              int dtype, void* workspace, size_t workspace_bytes, void* stream) {
    (void)workspace; (void)workspace_bytes;
    return svtad_conv_fwd_planned(x, nbr, w, bias, y, n, cin, cout, kk, tokens_per_batch, dtype, nullptr, stream);
}

extern "C" int svtad_conv_fwd_planned(const void* x, const int32_t* nbr, const void* w, const void* bias,
                                      void* y, int64_t n, int cin, int cout, int kk, int tokens_per_batch,
                                      int dtype, const void* plan, void* stream) {
    int rc = check_common("svtad_conv_fwd", n, cin, cout, kk, tokens_per_batch, dtype);
    if (rc) return rc;
    if (n == 0) return SVTAD_OK;
    SV_CHECK_ARG(x && nbr && w && y, "svtad_conv_fwd: null pointer");
    SV_CHECK_ARG(aligned(x, 16) && aligned(w, 16) && aligned(y, 16) && aligned(nbr, 16) && aligned(bias, 16),
                 "svtad_conv_fwd: x, nbr, w, bias and y must be 16-byte aligned");
    ConvArgs p{x, nbr, w, bias, y, n, cin, cout, kk, tokens_per_batch, dtype, plan};
    if (use_tc(SVTAD_OP_FWD, n, cin, cout, kk, dtype)) return tc_fwd(p, (cudaStream_t)stream);
    if (forced_path() == 2)
        return set_error(SVTAD_ERR_UNSUPPORTED, "svtad_conv_fwd: tensor-core path forced but shape/dtype unsupported");
    return simt_fwd(p, (cudaStream_t)stream);
}

static int conv_dgrad_planned(const void* gy, const int32_t* nbr, const void* w, void* gx, int64_t n, int cin, int cout,
                              int kk, int tokens_per_batch, int dtype, const void* plan, const int32_t* table_status,
                              void* workspace, size_t workspace_bytes, void* stream) {
    int rc = check_common("svtad_conv_dgrad", n, cin, cout, kk, tokens_per_batch, dtype);
    if (rc) return rc;
    if (n == 0) return SVTAD_OK;
    SV_CHECK_ARG(gy && nbr && w && gx, "svtad_conv_dgrad: null pointer");
    SV_CHECK_ARG(aligned(gy, 16) && aligned(w, 16) && aligned(gx, 16) && aligned(nbr, 16),
                 "svtad_conv_dgrad: gy, nbr, w and gx must be 16-byte aligned");
    if (cout % 4 != 0)
        return set_error(SVTAD_ERR_UNSUPPORTED, "svtad_conv_dgrad: C_out (%d) must be divisible by 4", cout);
    cudaStream_t s = (cudaStream_t)stream;
    ConvArgs p{gy, nbr, w, nullptr, gx, n, cin, cout, kk, tokens_per_batch, dtype, plan};
    if (use_tc(SVTAD_OP_DGRAD, n, cin, cout, kk, dtype)) {
        rc = tc_dgrad(p, table_status, s);
    } else {
        if (forced_path() == 2)
            return set_error(SVTAD_ERR_UNSUPPORTED, "svtad_conv_dgrad: tensor-core path forced but shape/dtype unsupported");
        rc = simt_dgrad_gather(p, table_status, s);
    }
    if (rc) return rc;
    if (table_status != nullptr) {
        // asymmetric tables: the scatter form runs instead (both kernels read the status word)
        size_t need = svtad_workspace_bytes(SVTAD_OP_DGRAD, n, cin, cout, kk, dtype);
        if (workspace == nullptr || workspace_bytes < need)
            return set_error(SVTAD_ERR_WORKSPACE, "svtad_conv_dgrad: workspace %zu < %zu bytes", workspace_bytes, need);
        rc = simt_dgrad_scatter(p, table_status, static_cast<float*>(workspace), s);
    }
    return rc;
}

extern "C" int svtad_conv_dgrad(const void* gy, const int32_t* nbr, const void* w, void* gx,
                                int64_t n, int cin, int cout, int kk, int tokens_per_batch,
                                int dtype, const int32_t* table_status, void* workspace,
                                size_t workspace_bytes, void* stream) {
    return conv_dgrad_planned(gy, nbr, w, gx, n, cin, cout, kk, tokens_per_batch, dtype, nullptr, table_status, workspace,
                              workspace_bytes, stream);
}

static int conv_wgrad_typed(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n, int cin,
                            int cout, int kk, int tokens_per_batch, int dtype, int grad_dtype, const void* plan,
                            void* workspace, size_t workspace_bytes, void* stream, bool fit = false) {
    int rc = check_common("svtad_conv_wgrad", n, cin, cout, kk, tokens_per_batch, dtype);
    if (rc) return rc;
    SV_CHECK_ARG(gw != nullptr, "svtad_conv_wgrad: gw is null");
    cudaStream_t s = (cudaStream_t)stream;
    if (n == 0) {
        SV_CUDA(cudaMemsetAsync(gw, 0, (size_t)kk * cin * cout * dtype_size(grad_dtype), s));
        if (gb) SV_CUDA(cudaMemsetAsync(gb, 0, (size_t)cout * dtype_size(grad_dtype), s));
        return SVTAD_OK;
    }
    SV_CHECK_ARG(gy && x && nbr, "svtad_conv_wgrad: null pointer");
    SV_CHECK_ARG(aligned(gy, 16) && aligned(x, 16) && aligned(gw, 16) && aligned(nbr, 16) && aligned(gb, 16),
                 "svtad_conv_wgrad: gy, x, nbr, gw and gb must be 16-byte aligned");
    SV_CHECK_ARG(workspace != nullptr && aligned(workspace, 256), "svtad_conv_wgrad: workspace is null or not 256-byte aligned");
    if (use_tc(SVTAD_OP_WGRAD, n, cin, cout, kk, dtype)) {
        if (plan != nullptr && pairs_wgrad_wanted(cin, kk))
            return pairs_wgrad(gy, x, plan, gw, gb, n, cin, cout, kk, dtype, grad_dtype, workspace, workspace_bytes, s);
        return tc_wgrad(gy, x, nbr, gw, gb, n, cin, cout, kk, tokens_per_batch, dtype, grad_dtype, workspace, workspace_bytes, fit, s);
    }
    if (forced_path() == 2)
        return set_error(SVTAD_ERR_UNSUPPORTED, "svtad_conv_wgrad: tensor-core path forced but shape/dtype unsupported");
    return simt_wgrad(gy, x, nbr, gw, gb, n, cin, cout, kk, tokens_per_batch, dtype, grad_dtype, workspace, workspace_bytes, s);
}

size_t svtad::wgrad_least_ws_bytes(int64_t n, int cin, int cout, int kk, int dtype, bool with_bias) {
    if (n <= 0 || cin <= 0 || cout <= 0 || kk <= 0) return 0;
    return use_tc(SVTAD_OP_WGRAD, n, cin, cout, kk, dtype) ? tc_wgrad_partials(1, with_bias, cin, cout, kk)
                                                           : simt_wgrad_ws_bytes(n, cin, cout, kk, dtype);
}

int svtad::conv_wgrad_fit(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb, int64_t n, int cin, int cout,
                          int kk, int tpb, int dtype, void* ws, size_t ws_bytes, cudaStream_t s) {
    return conv_wgrad_typed(gy, x, nbr, gw, gb, n, cin, cout, kk, tpb, dtype, dtype, nullptr, ws, ws_bytes, s, true);
}

extern "C" int svtad_conv_wgrad(const void* gy, const void* x, const int32_t* nbr, void* gw, void* gb,
                                int64_t n, int cin, int cout, int kk, int tokens_per_batch,
                                int dtype, void* workspace, size_t workspace_bytes, void* stream) {
    return conv_wgrad_typed(gy, x, nbr, gw, gb, n, cin, cout, kk, tokens_per_batch, dtype, dtype, nullptr, workspace,
                            workspace_bytes, stream);
}

extern "C" int svtad_conv_bwd(const void* gy, const void* x, const int32_t* nbr, const void* w, void* gx,
                              void* gw, void* gb, int64_t n, int cin, int cout, int kk,
                              int tokens_per_batch, int dtype, const int32_t* table_status,
                              void* workspace, size_t workspace_bytes, void* stream) {
    return svtad_conv_bwd_typed(gy, x, nbr, w, gx, gw, gb, n, cin, cout, kk, tokens_per_batch, dtype, dtype, nullptr, 0,
                                table_status, workspace, workspace_bytes, stream);
}

extern "C" int svtad_conv_bwd_typed(const void* gy, const void* x, const int32_t* nbr, const void* w, void* gx,
                                    void* gw, void* gb, int64_t n, int cin, int cout, int kk,
                                    int tokens_per_batch, int dtype, int grad_dtype, const void* plan,
                                    int plan_use, const int32_t* table_status, void* workspace,
                                    size_t workspace_bytes, void* stream) {
    return svtad_conv_bwd_planned(gy, x, nbr, w, gx, gw, gb, n, cin, cout, kk, tokens_per_batch, dtype, grad_dtype,
                                  const_cast<void*>(plan), plan_use, 0, table_status, workspace, workspace_bytes, stream);
}

extern "C" int svtad_conv_bwd_planned(const void* gy, const void* x, const int32_t* nbr, const void* w, void* gx,
                                      void* gw, void* gb, int64_t n, int cin, int cout, int kk,
                                      int tokens_per_batch, int dtype, int grad_dtype, void* plan, int plan_use,
                                      int plan_make, const int32_t* table_status, void* workspace,
                                      size_t workspace_bytes, void* stream) {
    SV_CHECK_ARG(grad_dtype == dtype || grad_dtype == SVTAD_F32,
                 "svtad_conv_bwd: weight gradients come in the features' type or in float32, not in type %d", grad_dtype);
    const void* rows_plan = plan_use & SVTAD_PLAN_ROWS ? plan : nullptr;
    const void* pairs_plan = plan_use & SVTAD_PLAN_PAIRS ? plan : nullptr;
    // Parts that are to be made first.  The lists alone go in front of the weight gradient on its stream.  With the row order
    // both come in one launch in front of the two kernels: made side by side, the lists are there first, the weight gradient
    // fills the GPU and the input gradient has to wait for it (4 720 rows, C = 768: a training pass 185 instead of 166 us).
    const int to_make = plan_make & ((gx != nullptr && rows_plan != nullptr ? SVTAD_PLAN_ROWS : 0) |
                                     (gw != nullptr && pairs_plan != nullptr ? SVTAD_PLAN_PAIRS : 0));
    auto make = [&](cudaStream_t on) {
        return to_make == 0 || n == 0 ? (int)SVTAD_OK : svtad_plan_build_parts(nbr, n, kk, tokens_per_batch, to_make, plan, on);
    };
    SV_CHECK_ARG(gx != nullptr || gw != nullptr, "svtad_conv_bwd: neither gx nor gw requested");
    SV_CHECK_ARG(gb == nullptr || gw != nullptr, "svtad_conv_bwd: gb needs gw");
    if (gw == nullptr) {
        if (int rc = make((cudaStream_t)stream)) return rc;
        return conv_dgrad_planned(gy, nbr, w, gx, n, cin, cout, kk, tokens_per_batch, dtype, rows_plan, table_status,
                                  workspace, workspace_bytes, stream);
    }
    if (gx == nullptr) {
        if (int rc = make((cudaStream_t)stream)) return rc;
        return conv_wgrad_typed(gy, x, nbr, gw, gb, n, cin, cout, kk, tokens_per_batch, dtype, grad_dtype, pairs_plan,
                                workspace, workspace_bytes, stream);
    }
    // workspace = [weight-gradient part | input-gradient part (scatter form, only with a status word)]
    const size_t w_part = svtad_bwd_workspace_bytes(n, cin, cout, kk, dtype, pairs_plan != nullptr ? plan_use : 0, 0);
    const size_t d_part = table_status != nullptr ? svtad_workspace_bytes(SVTAD_OP_DGRAD, n, cin, cout, kk, dtype) : 0;
    if (n > 0 && (workspace == nullptr || workspace_bytes < w_part + d_part))
        return set_error(SVTAD_ERR_WORKSPACE, "svtad_conv_bwd: workspace %zu < %zu bytes", workspace_bytes,
                         w_part + d_part);
    void* ws_d = d_part ? static_cast<char*>(workspace) + w_part : nullptr;
    cudaStream_t s = (cudaStream_t)stream;
    int dev = 0;
    SV_CUDA(cudaGetDevice(&dev));
    if (!overlap_backward() || n == 0 || dev >= MAX_DEVICES) {
        int rc = make(s);
        if (rc) return rc;
        rc = conv_wgrad_typed(gy, x, nbr, gw, gb, n, cin, cout, kk, tokens_per_batch, dtype, grad_dtype, pairs_plan,
                                  workspace, w_part, s);
        if (rc) return rc;
        return conv_dgrad_planned(gy, nbr, w, gx, n, cin, cout, kk, tokens_per_batch, dtype, rows_plan, table_status, ws_d,
                                  d_part, s);
    }
    SideLane& lane = g_lane[dev];
    std::lock_guard<std::mutex> hold(lane.mu);
    int rc = lane_ready(lane);
    if (rc) return rc;
    // The two kernels share the GPU.  While one of them cannot fill it, each is planned for half of it (unless the caller's
    // hint already says more): 8 084 rows, C = 256 (9.5 GFLOP a pass): 30 us against 32.5 planned for all of it.  From 18
    // GFLOP on both are planned for all of it and the second moves in as the first one's CTAs leave: 6 132 rows, C = 1024:
    // 249 -> 200 us; 3 744 rows, C = 320, 5x5: 74 -> 59 us.  With pair lists both are persistent and balanced over all SMs.
    const bool whole_gpu = pairs_plan != nullptr || 2.0 * (double)n * kk * cin * cout >= 18e9;
    struct FloorGuard {
        int old;
        explicit FloorGuard(int floor) : old(tc_set_share_floor(floor)) {}
        ~FloorGuard() { tc_set_share_floor(old); }
    } floor_guard(whole_gpu ? 1 : 2);
    if (to_make & SVTAD_PLAN_ROWS) {
        rc = make(s);
        if (rc) return rc;
    }
    // fork: the side stream starts where the caller's stream stands
    SV_CUDA(cudaEventRecord(lane.fork, s));
    SV_CUDA(cudaStreamWaitEvent(lane.stream, lane.fork, 0));
    int rc_w = SVTAD_OK, rc_d = SVTAD_OK;
    auto wgrad = [&] {
        rc_w = conv_wgrad_typed(gy, x, nbr, gw, gb, n, cin, cout, kk, tokens_per_batch, dtype, grad_dtype, pairs_plan, workspace,
                                w_part, lane.stream);
    };
    if (pairs_plan == nullptr) wgrad();
    else if (to_make == SVTAD_PLAN_PAIRS) rc_w = make(lane.stream);
    rc_d = conv_dgrad_planned(gy, nbr, w, gx, n, cin, cout, kk, tokens_per_batch, dtype, rows_plan, table_status, ws_d, d_part, s);
    if (pairs_plan != nullptr && rc_w == SVTAD_OK) wgrad();
    // join, also after an error: whatever was launched on the side stream is ordered before the caller's next work
    cudaError_t e1 = cudaEventRecord(lane.join, lane.stream);
    cudaError_t e2 = cudaStreamWaitEvent(s, lane.join, 0);
    if (rc_w) return rc_w;
    if (rc_d) return rc_d;
    if (e1 != cudaSuccess || e2 != cudaSuccess)
        return set_error(SVTAD_ERR_CUDA, "svtad_conv_bwd: joining the side stream failed: %s",
                         cudaGetErrorString(e1 != cudaSuccess ? e1 : e2));
    return SVTAD_OK;
}
