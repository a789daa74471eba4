// Python extension `_native`: the host path of the module and of the table functions in C++.
//
// A training step of one layer at a few thousand rows keeps the GPU busy for 30-50 us, while the same step driven by
// a Python autograd.Function over ctypes took 190-260 us of host time (argument checks, weak dictionaries, two Python
// frames of the autograd engine, a weight-gradient plan computed from scratch, one tensor.empty after the other):
// the GPU waited for the host.  Here a call is one extension function: shape checks, output allocation from torch's
// caching allocator, the library call, and - when a gradient is wanted - one autograd node whose apply() makes the
// library's one-call backward without touching the interpreter.
//
// What is known about a neighbor table (symmetric by construction, indices local to a batch row or not, the device
// status word of svtad_table_check, an int32 copy, how many of its entries are there) is kept per tensor object and
// version; entries of dead tables are swept as new tables are entered.  A table's work plan is not: a table can be
// written to without its version moving (a replayed graph that holds the selection, the C ABI, a raw pointer), so a
// layer makes its plan from what the table holds when its kernels run, every time.
#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <cstdlib>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "../../include/svtad.h"

namespace {

using at::Tensor;

void check(int rc) {
    if (rc == SVTAD_OK) return;
    const char* msg = svtad_last_error_string();
    if (rc == SVTAD_ERR_ARG || rc == SVTAD_ERR_UNSUPPORTED) TORCH_CHECK_VALUE(false, msg);
    TORCH_CHECK(false, "libsvtad error ", rc, ": ", msg);
}

void require_cuda(const Tensor& t) {
    TORCH_CHECK_VALUE(!t.defined() || t.is_cuda(), "SparseConv2D tensors must live on a CUDA device (there is no CPU path)");
}

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return SVTAD_F32;
        case at::kBFloat16: return SVTAD_BF16;
        case at::kHalf: return SVTAD_F16;
        default: TORCH_CHECK_VALUE(false, "unsupported dtype ", t, "; expected float32, bfloat16 or float16");
    }
}

Tensor empty_on(at::IntArrayRef sizes, at::ScalarType dtype, at::Device dev) {
    return Tensor(at::detail::empty_cuda(sizes, dtype, dev, std::nullopt));
}

void* stream_of(at::Device dev) { return static_cast<void*>(c10::cuda::getCurrentCUDAStream(dev.index()).stream()); }

// contiguous and 16-byte aligned (a contiguous slice of a larger tensor may start anywhere)
Tensor c16(const Tensor& t) {
    Tensor c = t.contiguous();
    if (c.numel() && reinterpret_cast<uintptr_t>(c.const_data_ptr()) % 16) c = c.clone();
    return c;
}

const void* ptr(const Tensor& t) { return t.defined() && t.numel() ? t.const_data_ptr() : nullptr; }
void* mptr(Tensor& t) { return t.defined() && t.numel() ? t.data_ptr() : nullptr; }
const int32_t* iptr(const Tensor& t) { return static_cast<const int32_t*>(ptr(t)); }

// ------------------------------------------------------------------------------------------------ table facts
// Another thread may be capturing a graph in the mode that forbids calls like these everywhere.
struct AnyCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    AnyCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
    ~AnyCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
};
bool landed(cudaEvent_t e) {
    AnyCapture relaxed;
    if (cudaEventQuery(e) == cudaSuccess) return true;
    (void)cudaGetLastError();
    return false;
}

// Landing places in pinned memory for a table's status word on its way to the host: one block, allocated at the first
// use (pinning memory takes milliseconds, so not once per table).  A place takes one copy: it is given back when its table
// dies or asks anew, and handed out again only after that copy has landed.  When all are taken the caller does without.
class HostWords {
  public:
    struct Place {
        volatile int32_t* word = nullptr;
        cudaEvent_t copied = nullptr;
    };
    bool take(Place& p) {
        std::lock_guard<std::mutex> hold(mu_);
        if (!page_ && !make_page()) return false;
        for (size_t i = 0; i < free_.size(); ++i) {
            if (!landed(free_[i].copied)) continue;
            p = free_[i];
            free_[i] = free_.back();
            free_.pop_back();
            return true;
        }
        return false;
    }
    void give_back(const Place& p) {
        std::lock_guard<std::mutex> hold(mu_);
        free_.push_back(p);
    }

  private:
    bool make_page() {
        AnyCapture relaxed;
        constexpr int PLACES = 128, BYTES = 256;
        if (cudaHostAlloc(&page_, PLACES * BYTES, cudaHostAllocPortable) != cudaSuccess) {
            (void)cudaGetLastError();
            page_ = nullptr;
            return false;
        }
        for (int i = 0; i < PLACES; ++i) {
            Place p;
            p.word = reinterpret_cast<volatile int32_t*>(static_cast<char*>(page_) + BYTES * i);
            if (cudaEventCreateWithFlags(&p.copied, cudaEventDisableTiming) == cudaSuccess) free_.push_back(p);
        }
        return true;
    }
    std::mutex mu_;
    void* page_ = nullptr;
    std::vector<Place> free_;
};
HostWords& host_words(int device) {      // an event belongs to the device it was made on, so one set per device
    constexpr int DEVICES = 64;
    static HostWords* h = new HostWords[DEVICES];
    return h[device % DEVICES];
}

// What svtad_table_check found for rows of kk taps and a tokens_per_batch.  The word on the device belongs to the stream it
// was written on: other streams neither wait for it nor keep its memory, so they ask for themselves.
struct Check {
    const int kk, device;
    const int64_t tpb;
    void* const stream;
    Tensor word;
    HostWords::Place host;       // where its copy on the host arrives, if there was a place
    Check(int kk_, int64_t tpb_, void* stream_, int device_) : kk(kk_), device(device_), tpb(tpb_), stream(stream_) {}
    ~Check() {
        if (host.word) host_words(device).give_back(host);
    }
};
constexpr size_t MOST_KEPT = 8;      // forms of one table kept at a time

struct Facts {
    c10::weak_intrusive_ptr<c10::TensorImpl> owner;
    int64_t version;
    int device;
    bool symmetric = false;      // by construction, or vouched for by the caller, ...
    int64_t symmetric_kk = 0;    // ... as rows of that many taps (0: not said)
    bool built = false;          // by this package: also batch-global over all of its rows
    int64_t local_n = -1;        // rows per batch row the answer `local` belongs to (-1: not asked yet)
    bool local = false;
    std::vector<std::shared_ptr<Check>> checks;      // one per reading of the table and stream, the newest last
    std::vector<std::pair<void*, Tensor>> i32;       // per stream, a contiguous, aligned int32 form of a table of another kind
    double density = -1;         // pairs per row and tap, as far as the host knows (only speed hangs on it)
    std::mutex mu;               // guards everything below `version`

    static int64_t version_of(const Tensor& t) { return t.is_inference() ? -1 : static_cast<int64_t>(t._version()); }
    explicit Facts(const Tensor& t) : owner(t.getIntrusivePtr()), version(version_of(t)), device(t.get_device()) {}
};

class FactStore {
  public:
    // facts of this very tensor object at its present version, entered if `make`; null otherwise.  Tensors made in
    // inference mode have no version counter, so only what speed hangs on can be remembered about them (`hint`).
    std::shared_ptr<Facts> find(const Tensor& t, bool make, bool hint = false) {
        if (t.is_inference() && !hint) return nullptr;
        std::lock_guard<std::mutex> hold(mu_);
        auto it = map_.find(t.unsafeGetTensorImpl());
        if (it != map_.end()) {
            if (!it->second->owner.expired() && it->second->version == Facts::version_of(t)) return it->second;
            map_.erase(it);
        }
        if (!make) return nullptr;
        // dead tables' entries go a few at a time: all of them while the tables are few, at the same cost where there are many
        auto e = map_.upper_bound(swept_);
        for (int i = 0; i < 8 && !map_.empty(); ++i) {
            if (e == map_.end()) e = map_.begin();
            swept_ = e->first;
            e = e->second->owner.expired() ? map_.erase(e) : std::next(e);
        }
        auto f = std::make_shared<Facts>(t);
        map_[t.unsafeGetTensorImpl()] = f;
        return f;
    }

  private:
    std::mutex mu_;
    const c10::TensorImpl* swept_ = nullptr;
    std::map<const c10::TensorImpl*, std::shared_ptr<Facts>, std::less<>> map_;
};

FactStore& store() {
    static FactStore* s = new FactStore;      // never destroyed: it may hold CUDA objects at exit
    return *s;
}

void mark_symmetric(const Tensor& t, bool built, double density = -1) {
    auto f = store().find(t, true, density >= 0);
    if (!f) return;
    std::lock_guard<std::mutex> hold(f->mu);
    if (density >= 0) f->density = density;
    if (t.is_inference()) return;
    f->symmetric = true;
    f->symmetric_kk = t.dim() > 1 ? t.size(-1) : 0;
    f->built = built;
}

// the table's density, where it or the tensor it looks into has one
double density_of(const Tensor& t) {
    auto known = [](const Tensor& u) {
        auto f = store().find(u, false, true);
        if (!f) return -1.0;
        std::lock_guard<std::mutex> hold(f->mu);
        return f->density;
    };
    const double d = known(t);
    return d >= 0 || !t.is_view() ? d : known(Tensor(at::TensorBase(t._base())));
}

// Expected pairs per row and tap of a table whose segments of `len` tokens, of an h x w grid per slice, keep k each.
double expected_density(int64_t len, int64_t k, int64_t h, int64_t w, int64_t ksize) {
    if (ksize < 1 || h < 1 || w < 1) return -1;
    const double share = len > 1 ? static_cast<double>(k - 1) / static_cast<double>(len - 1) : 0;
    double inside = 0;      // neighbors that lie on the grid, per token
    for (int64_t d = -(ksize / 2); d <= ksize / 2; ++d)
        for (int64_t e = -(ksize / 2); e <= ksize / 2; ++e)
            if (d != 0 || e != 0)
                inside += static_cast<double>(std::max<int64_t>(0, h - std::abs(d)) * std::max<int64_t>(0, w - std::abs(e))) / static_cast<double>(h * w);
    return (1 + inside * share) / static_cast<double>(ksize * ksize);
}
// ... and of a table of that density, n_prev rows per batch row, of which k are kept
double pruned_density(double density, int64_t kk, int64_t n_prev, int64_t k) {
    if (density < 0 || kk < 1) return -1;
    const double share = n_prev > 1 ? static_cast<double>(k - 1) / static_cast<double>(n_prev - 1) : 0;
    return (1 + std::max(0.0, density * static_cast<double>(kk) - 1) * share) / static_cast<double>(kk);
}

// the table's own facts or, for a view, those of the tensor it looks into
std::shared_ptr<Facts> symmetric_facts(const Tensor& t) {
    auto f = store().find(t, false);
    if (f && f->symmetric) return f;
    if (t.is_view()) {
        const at::TensorBase& b = t._base();
        const Tensor base = Tensor(at::TensorBase(b));
        f = store().find(base, false);
        if (f && f->symmetric) return f;
    }
    return nullptr;
}

bool is_known_symmetric(const Tensor& t, int64_t kk) {
    auto f = symmetric_facts(t);
    return f && (kk == 0 || f->symmetric_kk == 0 || f->symmetric_kk == kk);
}

bool capturing(void* stream) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(static_cast<cudaStream_t>(stream), &st) != cudaSuccess || st != cudaStreamCaptureStatusNone;
}

Tensor table_check(const Tensor& nbr, int64_t n, int kk, int64_t tpb, void* stream) {
    Tensor status = empty_on({1}, at::kInt, nbr.device());
    check(svtad_table_check(iptr(nbr), n, kk, static_cast<int>(tpb), static_cast<int32_t*>(status.data_ptr()), stream));
    return status;
}

std::shared_ptr<Check> kept_check(Facts& f, int kk, int64_t tpb, void* stream) {
    for (const auto& c : f.checks)
        if (c->kk == kk && c->tpb == tpb && c->stream == stream) return c;
    return nullptr;
}

// What the backward needs to know about a table: an undefined tensor when its entries are known to be symmetric (no
// validation, no scatter-form fallback), else the status word on the device.  The word is copied to the host behind
// the check, see found_symmetric().  Under graph capture the check belongs to the call: its word is written when the graph
// runs, in the graph's own memory.
Tensor status_for(const Tensor& table, const Tensor& nbr, int64_t n, int kk, int64_t tpb, void* stream) {
    if (tpb == 0 && is_known_symmetric(table, kk)) return Tensor();
    auto f = capturing(stream) ? nullptr : store().find(table, true);
    if (!f) return table_check(nbr, n, kk, tpb, stream);
    std::lock_guard<std::mutex> hold(f->mu);
    if (auto c = kept_check(*f, kk, tpb, stream)) return c->word;
    auto c = std::make_shared<Check>(kk, tpb, stream, f->device);
    c->word = table_check(nbr, n, kk, tpb, stream);
    if (host_words(f->device).take(c->host)) {
        C10_CUDA_CHECK(cudaMemcpyAsync(const_cast<int32_t*>(c->host.word), c->word.const_data_ptr(), sizeof(int32_t),
                                       cudaMemcpyDeviceToHost, static_cast<cudaStream_t>(stream)));
        C10_CUDA_CHECK(cudaEventRecord(c->host.copied, static_cast<cudaStream_t>(stream)));
    }
    if (f->checks.size() >= MOST_KEPT) f->checks.erase(f->checks.begin());
    f->checks.push_back(c);
    return c->word;
}

// Whether the validation pass of a table has come back clean.  Never waits: while the word's copy is under way the
// answer is no and the kernels read the word on the device.  By the time a network's backward reaches the layer the
// copy has arrived, and the fallback's three launches per backward go away.
bool found_symmetric(const Tensor& table, int kk, int64_t tpb, void* stream) {
    auto f = capturing(stream) ? nullptr : store().find(table, false);
    if (!f) return false;
    std::lock_guard<std::mutex> hold(f->mu);
    const auto c = kept_check(*f, kk, tpb, stream);
    return c && c->host.word && landed(c->host.copied) && *c->host.word == 0;
}

// A table of another kind is converted once per stream, and again in every captured call.
Tensor int32_table(const Tensor& table, void* stream) {
    if (table.scalar_type() == at::kInt && table.is_contiguous() &&
        (table.numel() == 0 || reinterpret_cast<uintptr_t>(table.const_data_ptr()) % 16 == 0))
        return table;
    auto f = capturing(stream) ? nullptr : store().find(table, true);
    if (!f) return c16(table.to(at::kInt));
    std::lock_guard<std::mutex> hold(f->mu);
    for (const auto& [on, form] : f->i32)
        if (on == stream) return form;
    Tensor form = c16(table.to(at::kInt));
    if (f->i32.size() >= MOST_KEPT) f->i32.erase(f->i32.begin());
    f->i32.emplace_back(stream, form);
    return form;
}

// Which parts of a work plan a layer's backward should use, of those that it has kernels for (`kernels`: 0 without a
// backward), and whether its forward should use one: only where the table's density is known, which for a caller's table
// means that this call, as one that reads the indices' kind from the values (see tokens_per_batch), may ask the device; once
// per table, and only for layers that a sparse table would bring a plan.  So the kernels that run, and with them the order of
// their sums, do not hang on when an answer arrives.  Nor does the forward's output hang on whether there is a backward: up to
// 74 tiles, where the forward without a plan may split a tile's K steps and give other bits, it goes by what a forward gains
// alone; beyond, where a row's sum is the same either way, it also uses a plan that the input gradient needs anyway.
struct Parts {
    int backward = 0;
    bool forward = false;
};
Parts plan_parts(const Tensor& table, int64_t n, int cin, int cout, int kk, int code, int kernels, bool may_ask, void* stream) {
    if (!svtad_plan_wanted(n, cin, cout, kk, code, 0.0)) return {};
    double density = density_of(table);
    if (density < 0 && may_ask && !capturing(stream)) {
        if (auto f = store().find(table, true)) {
            density = static_cast<double>(at::ge(table, 0).sum().item<int64_t>()) / static_cast<double>(table.numel());
            std::lock_guard<std::mutex> hold(f->mu);
            f->density = density;
        }
    }
    if (density < 0) return {};
    Parts p;
    p.backward = svtad_plan_wanted(n, cin, cout, kk, code, density) & kernels;
    p.forward = (p.backward & SVTAD_PLAN_ROWS && n > 74 * 128) || svtad_plan_wanted_fwd(n, cin, cout, kk, code, density);
    return p;
}

// tokens_per_batch of a call on [B, N, C] features: N when the table's indices are local to each batch row, else 0.
// Reference heuristic (sparse_conv_layer.py:170-177): local iff max(table) < N.  It needs the table's values, so it is
// evaluated once per table object; with one batch row the two readings agree, and a table this package built over all
// the rows is batch-global, so neither asks the device.
int64_t tokens_per_batch(const Tensor& table, int64_t B, int64_t N, int kk, int local) {
    if (B == 1 || N == 0) return 0;
    if (local >= 0) return local ? N : 0;
    if (table.numel() == 0) return 0;
    auto s = symmetric_facts(table);
    if (s && s->built && table.is_contiguous() && table.numel() == B * N * kk) {
        auto owner = s->owner.lock();
        if (owner && owner->numel() == table.numel()) return 0;
    }
    auto f = store().find(table, true);
    if (f) {
        std::lock_guard<std::mutex> hold(f->mu);
        if (f->local_n == N) return f->local ? N : 0;
    }
    const bool is_local = table.max().item<int64_t>() < N;
    if (f) {
        std::lock_guard<std::mutex> hold(f->mu);
        f->local_n = N;
        f->local = is_local;
    }
    return is_local ? N : 0;
}

// ------------------------------------------------------------------------------------------------ layer
struct Dims {
    int64_t n, tpb;
    int cin, cout, kk;
};

void require_shapes(const char* who, const Dims& d, const Tensor& nbr, const Tensor& bias) {
    TORCH_CHECK_VALUE(nbr.numel() == d.n * d.kk, who, ": neighbor table has ", nbr.numel(), " entries, expected ", d.n,
                      " rows x ", d.kk, " taps");
    TORCH_CHECK_VALUE(!bias.defined() || bias.numel() == d.cout, who, ": bias has ", bias.numel(), " elements, expected ", d.cout);
}

struct SparseConvBackward : public torch::autograd::Node {
    torch::autograd::SavedVariable x, table, weight;     // weight as it was used (the low-precision copy under autocast)
    Dims d;
    at::ScalarType w_dtype, b_dtype;                     // of the parameters
    Tensor status;
    Tensor plan;                                         // the forward's, with its row order; undefined without one
    int parts = 0;                                       // of a plan that the backward uses; it makes what the forward has not
    bool released = false;

    std::string name() const override { return "SparseConv2dBackward"; }

    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        x.reset_data();
        table.reset_data();
        weight.reset_data();
        plan.reset();
        released = true;
    }

    torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
        torch::autograd::variable_list out(3);
        if (!grads[0].defined()) return out;
        std::lock_guard<std::mutex> lock(mutex_);
        TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
        at::NoGradGuard no_grad;
        const bool need_x = task_should_compute_output(0), need_b = task_should_compute_output(2);
        const bool need_w = task_should_compute_output(1) || need_b;
        if (!need_x && !need_w) return out;
        auto self = getptr();
        Tensor xs = x.unpack(self), ts = table.unpack(self), w = weight.unpack(self);
        const Tensor gy = c16(grads[0]), xc = c16(xs), wc = c16(w), nbr = int32_table(ts, stream_of(ts.device()));
        const at::ScalarType dt = xc.scalar_type();
        TORCH_CHECK_VALUE(gy.scalar_type() == dt && wc.scalar_type() == dt, "grad_output, x and weight must share one dtype");
        TORCH_CHECK_VALUE(gy.numel() == d.n * d.cout, "grad_output has ", gy.numel(), " elements, expected ", d.n, " x ", d.cout);
        const at::Device dev = gy.device();
        c10::cuda::OptionalCUDAGuard guard(dev);
        void* stream = stream_of(dev);
        const int code = dtype_code(dt);
        // fp32 masters of a 16-bit layer get their gradient in fp32 straight from the kernel that sums it up
        const bool wide = dt != at::kFloat && w_dtype == at::kFloat && (!need_b || b_dtype == at::kFloat);
        const at::ScalarType gdt = wide ? at::kFloat : dt;
        Tensor gx, gw, gb, ws, st;
        if (need_x) {
            gx = empty_on(xs.sizes(), dt, dev);
            if (status.defined() && !found_symmetric(ts, d.kk, d.tpb, stream)) st = status;
        }
        if (need_w) gw = empty_on({d.kk, d.cin, d.cout}, gdt, dev);
        if (need_b) gb = empty_on({d.cout}, gdt, dev);
        const int use = parts & ((need_x ? SVTAD_PLAN_ROWS : 0) | (need_w ? SVTAD_PLAN_PAIRS : 0));
        const int make = use & ~(plan.defined() ? SVTAD_PLAN_ROWS : 0);
        Tensor pl = plan;
        const size_t bytes = need_w ? svtad_bwd_workspace_bytes(d.n, d.cin, d.cout, d.kk, code, use, st.defined())
                                    : (st.defined() ? svtad_workspace_bytes(SVTAD_OP_DGRAD, d.n, d.cin, d.cout, d.kk, code) : 0);
        if (bytes) ws = empty_on({static_cast<int64_t>(bytes)}, at::kByte, dev);
        if (make && !pl.defined()) pl = empty_on({static_cast<int64_t>(svtad_plan_bytes(d.n, d.kk))}, at::kByte, dev);
        check(svtad_conv_bwd_planned(ptr(gy), ptr(xc), iptr(nbr), ptr(wc), mptr(gx), mptr(gw), mptr(gb), d.n, d.cin, d.cout,
                                     d.kk, static_cast<int>(d.tpb), code, dtype_code(gdt), pl.defined() ? mptr(pl) : nullptr, use,
                                     make, iptr(st), mptr(ws), bytes, stream));
        out[0] = gx;
        if (task_should_compute_output(1)) out[1] = gw.scalar_type() == w_dtype ? gw : gw.to(w_dtype);
        if (need_b) out[2] = gb.scalar_type() == b_dtype ? gb : gb.to(b_dtype);
        return out;
    }
};

// The node below has no forward-mode formula: refused, as a torch.autograd.Function without jvp is.
void refuse_tangent(const Tensor& t) {
    TORCH_CHECK_NOT_IMPLEMENTED(!t.defined() || !t._fw_grad(/*level=*/0).defined(),
                                "SparseConv2d does not support forward mode automatic differentiation");
}

// weight_c / bias_c: the parameters in the computing dtype (the parameters themselves when it is theirs)
Tensor conv(Tensor x, const Tensor& table, const Tensor& weight, const Tensor& bias, const Tensor& weight_c,
            const Tensor& bias_c, int local) {
    require_cuda(x);
    require_cuda(table);
    require_cuda(weight_c);
    require_cuda(bias_c);
    refuse_tangent(x);
    refuse_tangent(weight);
    refuse_tangent(bias);
    const at::ScalarType dt = weight_c.scalar_type();
    if (x.scalar_type() != dt) x = x.to(dt);          // autocast: recorded by autograd like any cast
    const int code = dtype_code(dt);
    TORCH_CHECK_VALUE(!bias_c.defined() || bias_c.scalar_type() == dt, "x, weight and bias must share one dtype");
    Dims d;
    d.kk = static_cast<int>(weight_c.size(0));
    d.cin = static_cast<int>(weight_c.size(1));
    d.cout = static_cast<int>(weight_c.size(2));
    const bool batched = x.dim() == 3;
    d.n = x.numel() / d.cin;
    TORCH_CHECK_VALUE(d.n * d.cin == x.numel() && (!batched || x.size(2) == d.cin), "features do not have ", d.cin, " channels");
    const at::Device dev = x.device();
    c10::cuda::OptionalCUDAGuard guard(dev);
    void* stream = stream_of(dev);
    const bool grad = at::GradMode::is_enabled() &&
                      (x.requires_grad() || weight.requires_grad() || (bias.defined() && bias.requires_grad()));
    Tensor y, nbr, status, plan;
    Parts parts;
    {
        at::NoGradGuard no_grad;
        d.tpb = batched ? tokens_per_batch(table, x.size(0), x.size(1), d.kk, local) : 0;
        nbr = int32_table(table, stream);
        require_shapes("conv_fwd", d, nbr, bias_c);
        const Tensor xc = c16(x), wc = c16(weight_c), bc = bias_c.defined() ? c16(bias_c) : Tensor();
        if (batched) {
            y = empty_on({x.size(0), x.size(1), d.cout}, dt, dev);
        } else {
            y = empty_on({d.n, d.cout}, dt, dev);
        }
        if (grad && x.requires_grad()) status = status_for(table, nbr, d.n, d.kk, d.tpb, stream);
        const int kernels = !grad ? 0 : (x.requires_grad() ? SVTAD_PLAN_ROWS : 0) |
                            (weight.requires_grad() || (bias.defined() && bias.requires_grad()) ? SVTAD_PLAN_PAIRS : 0);
        parts = plan_parts(table, d.n, d.cin, d.cout, d.kk, code, kernels, batched && local < 0, stream);
        if (parts.forward) {
            plan = empty_on({static_cast<int64_t>(svtad_plan_bytes(d.n, d.kk))}, at::kByte, dev);
            check(svtad_plan_build_parts(iptr(nbr), d.n, d.kk, static_cast<int>(d.tpb), SVTAD_PLAN_ROWS, mptr(plan), stream));
        }
        check(svtad_conv_fwd_planned(ptr(xc), iptr(nbr), ptr(wc), ptr(bc), mptr(y), d.n, d.cin, d.cout, d.kk,
                                     static_cast<int>(d.tpb), code, ptr(plan), stream));
    }
    if (grad) {
        auto node = std::shared_ptr<SparseConvBackward>(new SparseConvBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(x, weight, bias));
        node->d = d;
        node->w_dtype = weight.scalar_type();
        node->b_dtype = bias.defined() ? bias.scalar_type() : dt;
        node->status = status;
        node->plan = plan;
        node->parts = parts.backward;
        node->x = torch::autograd::SavedVariable(x, false);
        node->table = torch::autograd::SavedVariable(table, false);
        node->weight = torch::autograd::SavedVariable(weight_c, false);
        torch::autograd::set_history(y, node);
    }
    return y;
}

// ------------------------------------------------------------------------------------------------ table functions
Tensor scores_of(const Tensor& scores) {
    require_cuda(scores);
    TORCH_CHECK_VALUE(scores.dim() == 2, "scores have ", scores.dim(), " dimensions, expected [segments, tokens]");
    return (scores.scalar_type() == at::kFloat ? scores : scores.to(at::kFloat)).contiguous();
}

Tensor table_init(int64_t B, int64_t T, int64_t h, int64_t w, int64_t ksize, at::Device dev) {
    c10::cuda::OptionalCUDAGuard guard(dev);
    Tensor out = empty_on({B, T * h * w, ksize * ksize}, at::kInt, dev);
    check(svtad_table_init(static_cast<int>(B), static_cast<int>(T), static_cast<int>(h), static_cast<int>(w),
                           static_cast<int>(ksize), static_cast<int32_t*>(mptr(out)), stream_of(dev)));
    mark_symmetric(out, true, expected_density(T * h * w, T * h * w, h, w, ksize));
    return out;
}

std::pair<Tensor, Tensor> table_build(const Tensor& scores_in, int64_t k, int64_t h, int64_t w, int64_t ksize) {
    const Tensor scores = scores_of(scores_in);
    const int64_t n_seg = scores.size(0), L = scores.size(1);
    const at::Device dev = scores.device();
    c10::cuda::OptionalCUDAGuard guard(dev);
    Tensor kept = empty_on({n_seg, k}, at::kInt, dev), table = empty_on({n_seg * k, ksize * ksize}, at::kInt, dev);
    check(svtad_table_build(static_cast<const float*>(ptr(scores)), static_cast<int>(n_seg), static_cast<int>(L),
                            static_cast<int>(k), static_cast<int>(h), static_cast<int>(w), static_cast<int>(ksize),
                            static_cast<int32_t*>(mptr(kept)), static_cast<int32_t*>(mptr(table)), stream_of(dev)));
    mark_symmetric(table, true, expected_density(L, k, h, w, ksize));
    return {kept, table};
}

Tensor topk_select(const Tensor& scores_in, int64_t k) {
    const Tensor scores = scores_of(scores_in);
    const int64_t B = scores.size(0), L = scores.size(1);
    const at::Device dev = scores.device();
    c10::cuda::OptionalCUDAGuard guard(dev);
    Tensor idx = empty_on({B, k}, at::kLong, dev);
    check(svtad_topk_select(static_cast<const float*>(ptr(scores)), static_cast<int>(B), static_cast<int>(L),
                            static_cast<int>(k), static_cast<int64_t*>(mptr(idx)), stream_of(dev)));
    return idx;
}

Tensor table_remap(const Tensor& table_in, const Tensor& idx_in, const Tensor& scratch_in) {
    require_cuda(table_in);
    require_cuda(idx_in);
    TORCH_CHECK_VALUE(table_in.dim() == 3, "the neighbor table has ", table_in.dim(), " dimensions, expected [batch, rows, taps]");
    auto sym = is_known_symmetric(table_in, table_in.size(2)) ? symmetric_facts(table_in) : nullptr;
    const Tensor table = int32_table(table_in, stream_of(table_in.device())), idx = idx_in.to(at::kLong).contiguous();
    const int64_t B = table.size(0), n_prev = table.size(1), kk = table.size(2), n_new = idx.size(1);
    const at::Device dev = table.device();
    c10::cuda::OptionalCUDAGuard guard(dev);
    Tensor scratch = scratch_in;
    if (!scratch.defined() || scratch.numel() < B * n_prev) scratch = empty_on({B * n_prev}, at::kInt, dev);
    Tensor out = empty_on({B, n_new, kk}, at::kInt, dev);
    check(svtad_table_remap(iptr(table), static_cast<const int64_t*>(ptr(idx)), static_cast<int>(B), static_cast<int>(n_prev),
                            static_cast<int>(n_new), static_cast<int>(kk), static_cast<int32_t*>(mptr(scratch)),
                            static_cast<int32_t*>(mptr(out)), stream_of(dev)));
    if (sym) mark_symmetric(out, sym->built, pruned_density(density_of(table_in), kk, n_prev, n_new));
    return out;
}

std::pair<Tensor, Tensor> table_select_remap(const Tensor& scores_in, const Tensor& table_in, int64_t k) {
    require_cuda(table_in);
    const Tensor scores = scores_of(scores_in);
    TORCH_CHECK_VALUE(table_in.dim() == 3, "the neighbor table has ", table_in.dim(), " dimensions, expected [batch, rows, taps]");
    auto sym = is_known_symmetric(table_in, table_in.size(2)) ? symmetric_facts(table_in) : nullptr;
    const Tensor table = int32_table(table_in, stream_of(table_in.device()));
    const int64_t B = table.size(0), n_prev = table.size(1), kk = table.size(2);
    TORCH_CHECK_VALUE(scores.dim() == 2 && scores.size(0) == B && scores.size(1) == n_prev, "table_select_remap: scores ",
                      scores.sizes(), " do not match the table's (", B, ", ", n_prev, ")");
    const at::Device dev = table.device();
    c10::cuda::OptionalCUDAGuard guard(dev);
    Tensor kept = empty_on({B, k}, at::kInt, dev), idx = empty_on({B, k}, at::kLong, dev), out = empty_on({B, k, kk}, at::kInt, dev);
    check(svtad_table_select_remap(static_cast<const float*>(ptr(scores)), iptr(table), static_cast<int>(B),
                                   static_cast<int>(n_prev), static_cast<int>(k), static_cast<int>(kk),
                                   static_cast<int32_t*>(mptr(kept)), static_cast<int64_t*>(mptr(idx)),
                                   static_cast<int32_t*>(mptr(out)), stream_of(dev)));
    if (sym) mark_symmetric(out, sym->built, pruned_density(density_of(table_in), kk, n_prev, k));
    return {idx, out};
}

// ------------------------------------------------------------------------------------------------ Python side
Tensor arg_tensor(PyObject* o, const char* name) {
    if (o == Py_None) return Tensor();
    TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a tensor");
    return THPVariable_Unpack(o);
}
Tensor need_tensor(PyObject* o, const char* name) {
    Tensor t = arg_tensor(o, name);
    TORCH_CHECK_TYPE(t.defined(), name, " must be a tensor");
    return t;
}
int64_t arg_int(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}
void arg_count(Py_ssize_t got, Py_ssize_t want, const char* who) {
    TORCH_CHECK_TYPE(got == want, who, ": expected ", want, " arguments, got ", got);
}
PyObject* pair(std::pair<Tensor, Tensor>&& p) {
    return PyTuple_Pack(2, py::reinterpret_steal<py::object>(THPVariable_Wrap(p.first)).ptr(),
                        py::reinterpret_steal<py::object>(THPVariable_Wrap(p.second)).ptr());
}

// conv(x, table, weight, bias, weight_c, bias_c, local): local = None (decide), True or False
PyObject* py_conv(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 7, "conv");
    const Tensor x = need_tensor(a[0], "x"), table = need_tensor(a[1], "neighbor_indices"), w = need_tensor(a[2], "weight"),
                 b = arg_tensor(a[3], "bias"), wc = need_tensor(a[4], "weight"), bc = arg_tensor(a[5], "bias");
    int local = -1;
    if (a[6] != Py_None) {
        local = PyObject_IsTrue(a[6]);
        if (local < 0) throw python_error();
    }
    Tensor y;
    {
        pybind11::gil_scoped_release no_gil;
        y = conv(x, table, w, b, wc, bc, local);
    }
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

PyObject* py_table_init(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 6, "table_init");
    return THPVariable_Wrap(table_init(arg_int(a[0]), arg_int(a[1]), arg_int(a[2]), arg_int(a[3]), arg_int(a[4]),
                                       at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(arg_int(a[5])))));
    END_HANDLE_TH_ERRORS
}

PyObject* py_table_build(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 5, "table_build");
    return pair(table_build(need_tensor(a[0], "scores"), arg_int(a[1]), arg_int(a[2]), arg_int(a[3]), arg_int(a[4])));
    END_HANDLE_TH_ERRORS
}

PyObject* py_topk_select(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 2, "topk_select");
    return THPVariable_Wrap(topk_select(need_tensor(a[0], "scores"), arg_int(a[1])));
    END_HANDLE_TH_ERRORS
}

PyObject* py_table_remap(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 3, "table_remap");
    return THPVariable_Wrap(table_remap(need_tensor(a[0], "table"), need_tensor(a[1], "idx"), arg_tensor(a[2], "scratch")));
    END_HANDLE_TH_ERRORS
}

PyObject* py_table_select_remap(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 3, "table_select_remap");
    return pair(table_select_remap(need_tensor(a[0], "scores"), need_tensor(a[1], "table"), arg_int(a[2])));
    END_HANDLE_TH_ERRORS
}

PyObject* py_mark_symmetric(PyObject*, PyObject* t) {
    HANDLE_TH_ERRORS
    mark_symmetric(need_tensor(t, "table"), false);
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

PyObject* py_is_known_symmetric(PyObject*, PyObject* t) {
    HANDLE_TH_ERRORS
    const Tensor table = need_tensor(t, "table");
    return PyBool_FromLong(is_known_symmetric(table, table.dim() > 1 ? table.size(-1) : 0));
    END_HANDLE_TH_ERRORS
}

// table_status(table, kk, tokens_per_batch): None for a table known to be symmetric, else the device status word
PyObject* py_table_status(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    arg_count(n, 3, "table_status");
    const Tensor table = need_tensor(a[0], "table");
    require_cuda(table);
    const int kk = static_cast<int>(arg_int(a[1]));
    c10::cuda::OptionalCUDAGuard guard(table.device());
    const Tensor nbr = int32_table(table, stream_of(table.device()));
    const Tensor st = status_for(table, nbr, nbr.numel() / kk, kk, arg_int(a[2]), stream_of(table.device()));
    if (!st.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(st);
    END_HANDLE_TH_ERRORS
}

#define FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FAST("conv", py_conv),
    FAST("table_init", py_table_init),
    FAST("table_build", py_table_build),
    FAST("topk_select", py_topk_select),
    FAST("table_remap", py_table_remap),
    FAST("table_select_remap", py_table_select_remap),
    FAST("table_status", py_table_status),
    {"mark_symmetric", py_mark_symmetric, METH_O, nullptr},
    {"is_known_symmetric", py_is_known_symmetric, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", "Host path of SparseConv2D over libsvtad.so.", -1, methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module_def); }
