// C ABI of einsums_gb300: argument checking, algorithm reporting, lowering of
// an arbitrary (C, A, B) index pattern to the canonical batched contraction,
// and dispatch to the kernels.  No exception crosses this file's entry points.
#include <algorithm>
#include <cmath>
#include <condition_variable>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/einsums_gb300/classify.hpp"
#include "common.cuh"

namespace eg {

namespace detail = ::einsums_gb300::detail;

namespace {
thread_local std::string g_last_error;
thread_local eg_split_report g_split_report = {0, 0, 0, 0.0};

// Library-wide registries are allocated once and never destroyed, so objects
// released during static destruction at process exit (cached plans, workspaces)
// never touch an already-destroyed container.
std::mutex &g_mem_mutex = *new std::mutex;
size_t g_budget = 0; // 0 = unlimited
size_t g_in_use = 0;
std::map<void *, size_t> &g_sizes = *new std::map<void *, size_t>;

struct WsKey {
    int dev;
    cudaStream_t stream;
    bool operator<(const WsKey &o) const { return dev != o.dev ? dev < o.dev : stream < o.stream; }
};
struct WsBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
};
std::mutex &g_ws_mutex = *new std::mutex;
std::map<WsKey, WsBuf> &g_ws = *new std::map<WsKey, WsBuf>;
} // namespace

void set_error(const std::string &msg) { g_last_error = msg; }

eg_status fail(eg_status st, const std::string &msg) {
    g_last_error = msg;
    return st;
}

eg_status cuda_fail(cudaError_t err, const char *what) {
    g_last_error = std::string(what) + ": " + cudaGetErrorName(err) + " (" + cudaGetErrorString(err) + ")";
    return err == cudaErrorMemoryAllocation ? EG_ERROR_OUT_OF_MEMORY : EG_ERROR_CUDA;
}

namespace {
eg_status malloc_once(size_t bytes, void **ptr) {
    std::lock_guard<std::mutex> lk(g_mem_mutex);
    if (g_budget && g_in_use + bytes > g_budget)
        return fail(EG_ERROR_OUT_OF_MEMORY, "device allocation of " + std::to_string(bytes) +
                                                " bytes exceeds the memory budget of " + std::to_string(g_budget));
    void *p = nullptr;
    cudaError_t err = cudaMalloc(&p, bytes ? bytes : 1);
    if (err != cudaSuccess) {
        if (err == cudaErrorMemoryAllocation) cudaGetLastError(); // not sticky: leave no trace for later checks
        return cuda_fail(err, "cudaMalloc");
    }
    g_sizes[p] = bytes;
    g_in_use += bytes;
    *ptr = p;
    return EG_SUCCESS;
}
} // namespace

// The scratch buffers of a device (ScratchLease).  Several, so that work waiting on one stream
// does not hold up another: a call takes the buffer that its stream used last, else one whose
// work is done, else a new one while all of them stay below kScratchTotal; only then does it
// wait on the GPU for another stream's work.
struct Scratch {
    void *ptr = nullptr;
    size_t bytes = 0;
    cudaEvent_t last = nullptr; // after the last lease's work
    cudaStream_t stream = nullptr;
    bool taken = false; // by a lease that has not ended
    bool fresh = false; // allocated, its header not yet cleared
    uint64_t turn = 0;
};

constexpr int kScratchBuffers = 8;
constexpr size_t kScratchTotal = size_t(5) << 30, kScratchUnit = size_t(64) << 20;
struct ScratchPool {
    std::mutex mu;
    std::condition_variable ended; // a lease
    Scratch buffers[kScratchBuffers];
    uint64_t turns = 0;
};

namespace {
std::mutex &g_scratch_mutex = *new std::mutex;
std::map<int, ScratchPool> &g_scratch = *new std::map<int, ScratchPool>;

bool done(const Scratch &x) { // the work of its last lease
    if (!x.last) return true;
    const cudaError_t err = cudaEventQuery(x.last);
    if (err == cudaErrorNotReady) cudaGetLastError();
    return err == cudaSuccess;
}

// Waits for the buffer's last user and frees it (not taken, its pool locked).
void drop_scratch(Scratch &x) {
    if (!x.ptr) return;
    RelaxedCapture relaxed;
    if (x.last) cudaEventSynchronize(x.last);
    tracked_free(x.ptr);
    x.ptr = nullptr;
    x.bytes = 0;
}

// Gives back every device's scratch; false when there was none.
bool trim_scratch() {
    std::vector<ScratchPool *> all;
    {
        std::lock_guard<std::mutex> lk(g_scratch_mutex);
        for (auto &kv : g_scratch) all.push_back(&kv.second);
    }
    bool any = false;
    for (ScratchPool *p : all) {
        std::unique_lock<std::mutex> lk(p->mu);
        for (Scratch &x : p->buffers) {
            p->ended.wait(lk, [&] { return !x.taken; });
            any |= x.ptr != nullptr;
            drop_scratch(x);
        }
    }
    return any;
}

// Whether `want` bytes can be allocated once `back` bytes have been freed: under the memory
// budget, and with a thirty-second of the device's memory left free.
bool scratch_fits(size_t want, size_t back) {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || free_b + back < want + total_b / 32) return false;
    std::lock_guard<std::mutex> lk(g_mem_mutex);
    return !g_budget || g_in_use + want <= g_budget + back;
}

// A buffer of at least `bytes` that is not taken (its pool locked), or null; `wait`: all that would
// do are taken, and one may come back.
Scratch *choose_scratch(ScratchPool &p, cudaStream_t s, size_t bytes, bool &wait) {
    Scratch *own = nullptr, *idle = nullptr, *busy = nullptr, *empty = nullptr, *small = nullptr;
    size_t held = 0;
    wait = false;
    for (Scratch &x : p.buffers) {
        held += x.bytes;
        if (x.taken) {
            wait |= x.bytes >= bytes;
        } else if (!x.ptr) {
            empty = &x;
        } else if (x.bytes < bytes) {
            if (!small || (x.stream == s) > (small->stream == s) ||
                ((x.stream == s) == (small->stream == s) && x.turn < small->turn))
                small = &x;
        } else if (x.stream == s) {
            if (!own || x.bytes < own->bytes) own = &x;
        } else if (done(x)) {
            if (!idle || x.bytes < idle->bytes) idle = &x;
        } else if (!busy || x.turn < busy->turn) {
            busy = &x;
        }
    }
    if (own) return own;
    if (idle) return idle;
    const size_t want = (bytes + kScratchUnit - 1) / kScratchUnit * kScratchUnit;
    auto allocate = [&](Scratch &x) -> Scratch * {
        if (malloc_once(want, &x.ptr) != EG_SUCCESS) {
            set_error("");
            return nullptr;
        }
        x.bytes = want;
        x.fresh = true;
        return &x;
    };
    // beside those that are too small: freeing one waits for all work on the device, which may be
    // held up, so that is left for when there is no other way
    if (empty && (held + want <= kScratchTotal || held == 0) && scratch_fits(want, 0)) {
        if (Scratch *x = allocate(*empty)) return x;
    }
    if (!busy && !wait && small && scratch_fits(want, small->bytes)) {
        drop_scratch(*small);
        return allocate(*small);
    }
    return busy;
}
} // namespace

bool drop_cached_plans(); // batched.cu

eg_status tracked_malloc(size_t bytes, void **ptr, bool make_room) {
    const eg_status st = malloc_once(bytes, ptr);
    if (st != EG_ERROR_OUT_OF_MEMORY || !make_room) return st;
    const bool scratch = trim_scratch(), plans = drop_cached_plans();
    if (!scratch && !plans) return st;
    set_error("");
    return malloc_once(bytes, ptr);
}

ScratchLease::ScratchLease(cudaStream_t s, size_t bytes) : s_(s) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    ScratchPool *p = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_scratch_mutex);
        p = &g_scratch[dev];
    }
    RelaxedCapture relaxed;
    std::unique_lock<std::mutex> lk(p->mu);
    Scratch *x = nullptr;
    for (bool wait = true; wait;) {
        x = choose_scratch(*p, s, bytes + kHeader, wait);
        if (x) break;
        if (wait) p->ended.wait(lk);
    }
    if (!x || (!x->last && cudaEventCreateWithFlags(&x->last, cudaEventDisableTiming) != cudaSuccess) ||
        cudaStreamWaitEvent(s, x->last, 0) != cudaSuccess ||
        (x->fresh && cudaMemsetAsync(x->ptr, 0, kHeader, s) != cudaSuccess)) {
        cudaGetLastError();
        return;
    }
    x->taken = true;
    x->fresh = false;
    x->stream = s;
    x->turn = ++p->turns;
    pool_ = p;
    buffer_ = x;
    ptr_ = (char *)x->ptr + kHeader;
}

ScratchLease::~ScratchLease() {
    if (!pool_) return;
    if (cudaEventRecord(buffer_->last, s_) != cudaSuccess) { // never leave the buffer unguarded
        cudaStreamSynchronize(s_);
        cudaGetLastError();
    }
    {
        std::lock_guard<std::mutex> lk(pool_->mu);
        buffer_->taken = false;
    }
    pool_->ended.notify_all();
}

eg_status tracked_free(void *ptr) {
    if (!ptr) return EG_SUCCESS;
    {
        std::lock_guard<std::mutex> lk(g_mem_mutex);
        auto it = g_sizes.find(ptr);
        if (it == g_sizes.end()) return fail(EG_ERROR_INVALID_ARGUMENT, "eg_device_free: pointer not from eg_device_alloc");
        g_in_use -= it->second;
        g_sizes.erase(it);
    }
    EG_CUDA(cudaFree(ptr));
    return EG_SUCCESS;
}

eg_status workspace(cudaStream_t stream, size_t bytes, void **ptr) {
    int dev = 0;
    EG_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_ws_mutex);
    WsBuf &b = g_ws[WsKey{dev, stream}];
    if (b.bytes < bytes) {
        if (b.ptr) {
            // Earlier work on this stream may still read the old buffer.
            EG_CUDA(cudaStreamSynchronize(stream));
            eg_status st = tracked_free(b.ptr);
            b.ptr = nullptr;
            b.bytes = 0;
            if (st != EG_SUCCESS) return st;
        }
        size_t want = std::max(bytes, b.bytes * 2);
        want = (want + 0xFFFFF) & ~size_t(0xFFFFF);
        eg_status st = tracked_malloc(want, &b.ptr);
        if (st != EG_SUCCESS) {
            b.ptr = nullptr;
            return st;
        }
        b.bytes = want;
    }
    *ptr = b.ptr;
    return EG_SUCCESS;
}

void set_split_report(const eg_split_report &r) { g_split_report = r; }

namespace {
std::mutex &g_status_mutex = *new std::mutex;
std::map<WsKey, int *> &g_status = *new std::map<WsKey, int *>;
} // namespace

// One status word per (device, stream), allocated on first use.  A stream that
// is being captured into a CUDA graph cannot allocate: it gets its own word if
// one exists, else the device's shared word for captured launches (created with
// the first word of the device, outside any capture).
eg_status status_word(cudaStream_t stream, int **ptr) {
    int dev = 0;
    EG_CUDA(cudaGetDevice(&dev));
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    EG_CUDA(cudaStreamIsCapturing(stream, &cap));
    std::lock_guard<std::mutex> lk(g_status_mutex);
    const WsKey shared_key{dev, reinterpret_cast<cudaStream_t>(~uintptr_t(0))};
    auto found = g_status.find(WsKey{dev, stream});
    if (found != g_status.end() && found->second) {
        *ptr = found->second;
        return EG_SUCCESS;
    }
    if (cap != cudaStreamCaptureStatusNone) {
        auto sh = g_status.find(shared_key);
        if (sh == g_status.end() || !sh->second)
            return fail(EG_ERROR_NOT_SUPPORTED, "first call of the library on this device is under stream capture");
        *ptr = sh->second;
        return EG_SUCCESS;
    }
    for (const WsKey &key : {shared_key, WsKey{dev, stream}}) {
        int *&w = g_status[key];
        if (w) continue;
        // (a stream of its own: the legacy one must not be used beside some captures)
        RelaxedCapture relaxed;
        cudaStream_t own = nullptr;
        int *fresh = nullptr;
        cudaError_t err = cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking);
        if (err == cudaSuccess) err = cudaMalloc(&fresh, 256);
        if (err == cudaSuccess) err = cudaMemsetAsync(fresh, 0, 256, own);
        if (err == cudaSuccess) err = cudaStreamSynchronize(own);
        if (own) cudaStreamDestroy(own);
        if (err != cudaSuccess) {
            if (fresh) cudaFree(fresh);
            cudaGetLastError(); // leave no trace for later checks
            return cuda_fail(err, "status word");
        }
        w = fresh;
    }
    *ptr = g_status[WsKey{dev, stream}];
    return EG_SUCCESS;
}

namespace {

using detail::Algorithm;
using detail::Labels;
using detail::View;

eg_status check_tensor(const eg_tensor *t, const int32_t *labels, const char *name) {
    if (!t) return fail(EG_ERROR_INVALID_ARGUMENT, std::string(name) + " is NULL");
    if (t->rank < 0 || t->rank > EG_MAX_RANK)
        return fail(EG_ERROR_RANK, std::string(name) + " has rank " + std::to_string(t->rank) + " (max 8)");
    if (t->rank > 0 && !labels) return fail(EG_ERROR_INVALID_ARGUMENT, std::string(name) + " labels are NULL");
    int64_t n = 1;
    for (int i = 0; i < t->rank; i++) {
        if (t->extent[i] < 0) return fail(EG_ERROR_DIMENSION, std::string(name) + " has a negative extent");
        if (t->stride[i] < 0) return fail(EG_ERROR_NOT_SUPPORTED, std::string(name) + " has a negative stride");
        n *= t->extent[i];
    }
    if (n > 0 && !t->data) return fail(EG_ERROR_INVALID_ARGUMENT, std::string(name) + " data is NULL");
    return EG_SUCCESS;
}

View view_of(const eg_tensor *t) {
    View v;
    v.rank = t->rank;
    for (int i = 0; i < t->rank; i++) {
        v.extent[i] = t->extent[i];
        v.stride[i] = t->stride[i];
    }
    return v;
}

Labels labels_of(const int32_t *l, int n) {
    Labels x;
    for (int i = 0; i < n; i++) x.push(l[i]);
    return x;
}

struct Mode {
    int64_t ext;
    int64_t s[3];
};

struct Modes {
    int n = 0;
    Mode m[2 * EG_MAX_RANK]; // summed indices of A alone and of B alone
};

// Sort by the given operand's stride (descending) and merge neighbours that
// are contiguous in all three operands.  False when more modes are left than a group holds
// (summed indices of A alone and of B alone may be sixteen).
bool fold(Modes &modes, int primary, ModeGroup &g) {
    auto before = [&](const Mode &a, const Mode &b) {
        if (a.s[primary] != b.s[primary]) return a.s[primary] > b.s[primary];
        for (int t = 0; t < 3; t++)
            if (a.s[t] != b.s[t]) return a.s[t] > b.s[t];
        return false;
    };
    for (int i = 1; i < modes.n; i++) { // (few: insertion, which keeps the order of equals)
        const Mode x = modes.m[i];
        int j = i;
        for (; j > 0 && before(x, modes.m[j - 1]); j--) modes.m[j] = modes.m[j - 1];
        modes.m[j] = x;
    }
    g = ModeGroup{};
    for (int i = 0; i < modes.n; i++) {
        const Mode &m = modes.m[i];
        if (m.ext == 1) continue; // extent-1 modes contribute nothing
        bool merge = g.n > 0;
        for (int t = 0; t < 3 && merge; t++) merge = g.s[t][g.n - 1] == m.s[t] * m.ext;
        if (!merge) {
            if (g.n == kMaxModes) return false;
            g.ext[g.n++] = 1;
        }
        g.ext[g.n - 1] *= m.ext;
        for (int t = 0; t < 3; t++) g.s[t][g.n - 1] = m.s[t];
        g.total *= m.ext;
    }
    return true;
}

struct Lowered {
    Contraction c;
    bool empty_c = false;
};

eg_status lower(const int32_t *Cl, const eg_tensor *C, const int32_t *Al, const eg_tensor *A, const int32_t *Bl,
                const eg_tensor *B, int semantics, Lowered &out) {
    struct U {
        int32_t label = 0;
        int64_t ext = -1;
        int64_t s[3] = {0, 0, 0};
        bool in[3] = {false, false, false};
    };
    U us[3 * EG_MAX_RANK];
    int count = 0;
    auto add = [&](const int32_t *labels, const eg_tensor *t, int which, const char *name) -> eg_status {
        for (int i = 0; i < t->rank; i++) {
            U *it = us;
            while (it != us + count && it->label != labels[i]) it++;
            if (it == us + count) us[count++].label = labels[i];
            if (it->ext >= 0 && it->ext != t->extent[i])
                return fail(EG_ERROR_DIMENSION, std::string("index ") + std::to_string(labels[i]) + " of " + name +
                                                    " has extent " + std::to_string(t->extent[i]) + " but " +
                                                    std::to_string(it->ext) + " elsewhere");
            it->ext = t->extent[i];
            it->s[which] += t->stride[i]; // repeated labels walk the diagonal (get_stride_for sums them)
            it->in[which] = true;
        }
        return EG_SUCCESS;
    };
    eg_status st;
    if ((st = add(Cl, C, 2, "C")) != EG_SUCCESS) return st;
    if ((st = add(Al, A, 0, "A")) != EG_SUCCESS) return st;
    if ((st = add(Bl, B, 1, "B")) != EG_SUCCESS) return st;

    Modes batch, m, n, k;
    auto put = [](Modes &to, const U &u) { to.m[to.n++] = Mode{u.ext, {u.s[0], u.s[1], u.s[2]}}; };
    int64_t c_elems = 1;
    for (int i = 0; i < count; i++) {
        const U &u = us[i];
        if (u.in[2]) c_elems *= u.ext;
        if (u.in[2] && u.in[0] && u.in[1])
            put(batch, u);
        else if (u.in[2] && u.in[1] && !u.in[0])
            put(n, u);
        else if (u.in[2])
            put(m, u); // in A only, or C-only broadcast (A stride 0)
        else if (u.in[0] && u.in[1])
            put(k, u);
        else if (semantics == EG_SEMANTICS_PYTHON)
            put(k, u); // operand-only index: summed over the unique-index space
        // else: C++ semantics hold an operand-only index at 0
    }
    // Repeated C labels address the diagonal only; the number of C positions
    // written is the product over unique labels, as in the reference loops.
    out.c = Contraction{};
    if (!fold(batch, 2, out.c.batch) || !fold(m, 0, out.c.m) || !fold(n, 1, out.c.n) || !fold(k, 0, out.c.k))
        return fail(EG_ERROR_NOT_SUPPORTED, "more than " + std::to_string(kMaxModes) + " separate indices in one role");
    out.c.A = A->data;
    out.c.B = B->data;
    out.c.C = C->data;
    out.c.c_elems = c_elems;
    out.empty_c = (c_elems == 0);
    return EG_SUCCESS;
}

Algorithm classify_labels(const detail::Analysis &an, int semantics) {
    return semantics == EG_SEMANTICS_PYTHON ? detail::classify_py(an) : detail::classify_cpp(an);
}

// The algorithm of a call: that of its pattern, or the generic one where the views or the
// options say so.
Algorithm choose(const detail::Analysis &an, Algorithm of_pattern, const eg_options &opt, const eg_tensor *C,
                 const eg_tensor *A, const eg_tensor *B) {
    const Algorithm alg = opt.only_generic ? Algorithm::GENERIC : of_pattern;
    return opt.semantics == EG_SEMANTICS_CPP ? detail::apply_vetoes(alg, an, view_of(C), view_of(A), view_of(B)) : alg;
}

} // namespace

// The algorithm the reference reports for a call (classification and stride
// vetoes), without running it.
eg_status classify_call(const int32_t *Cl, const eg_tensor *C, const int32_t *Al, const eg_tensor *A,
                        const int32_t *Bl, const eg_tensor *B, const eg_options *opt_in, int32_t *alg_out) {
    eg_options opt;
    eg_options_default(&opt);
    if (opt_in) opt = *opt_in;
    eg_status st;
    if ((st = check_tensor(C, Cl, "C")) != EG_SUCCESS) return st;
    if ((st = check_tensor(A, Al, "A")) != EG_SUCCESS) return st;
    if ((st = check_tensor(B, Bl, "B")) != EG_SUCCESS) return st;
    const detail::Analysis an(labels_of(Cl, C->rank), labels_of(Al, A->rank), labels_of(Bl, B->rank));
    const Algorithm alg = choose(an, classify_labels(an, opt.semantics), opt, C, A, B);
    *alg_out = (int32_t)alg;
    return EG_SUCCESS;
}

eg_status einsum_impl(double cp, const int32_t *Cl, const eg_tensor *C, double ab, const int32_t *Al, const eg_tensor *A,
                      const int32_t *Bl, const eg_tensor *B, const eg_options *opt_in, cudaStream_t stream,
                      int32_t *alg_out) {
    eg_options opt;
    eg_options_default(&opt);
    if (opt_in) opt = *opt_in;
    if (opt.semantics != EG_SEMANTICS_CPP && opt.semantics != EG_SEMANTICS_PYTHON)
        return fail(EG_ERROR_INVALID_ARGUMENT, "unknown semantics");
    if (opt.precision != EG_PRECISION_FP64 && opt.precision != EG_PRECISION_SPLIT_BF16)
        return fail(EG_ERROR_INVALID_ARGUMENT, "unknown precision");
    eg_status st;
    if ((st = check_tensor(C, Cl, "C")) != EG_SUCCESS) return st;
    if ((st = check_tensor(A, Al, "A")) != EG_SUCCESS) return st;
    if ((st = check_tensor(B, Bl, "B")) != EG_SUCCESS) return st;

    const detail::Analysis an(labels_of(Cl, C->rank), labels_of(Al, A->rank), labels_of(Bl, B->rank));
    const Algorithm alg = choose(an, classify_labels(an, opt.semantics), opt, C, A, B);
    if (alg_out) *alg_out = (int32_t)alg;

    Lowered low;
    if ((st = lower(Cl, C, Al, A, Bl, B, opt.semantics, low)) != EG_SUCCESS) return st;
    if (low.empty_c) return EG_SUCCESS;
    Contraction &c = low.c;
    c.cp = cp;
    c.ab = ab;
    // The C++ DOT and GER paths multiply C by C_prefactor instead of zeroing it
    // (Dispatch.hpp:907, :343-346), so a NaN in C survives C_prefactor == 0 there.
    c.zero_when_cp_zero = !(opt.semantics == EG_SEMANTICS_CPP && (alg == Algorithm::DOT || alg == Algorithm::GER));

    // A repeated C label addresses only C's diagonal; the prefactor still
    // applies to all of C first (BaseAlgebra.hpp:129-133, PyTensorAlgebra.hpp:541-563).
    bool c_repeats = false;
    for (int i = 0; i < C->rank; i++)
        for (int j = i + 1; j < C->rank; j++) c_repeats |= Cl[i] == Cl[j];
    if (c_repeats && !(c.cp == 1.0)) {
        ModeGroup cg;
        for (int i = 0; i < C->rank; i++) {
            cg.ext[cg.n] = C->extent[i];
            cg.s[2][cg.n] = C->stride[i];
            cg.total *= C->extent[i];
            cg.n++;
        }
        if ((st = launch_scale(cg, C->data, c.cp, stream)) != EG_SUCCESS) return st;
        c.cp = 1.0;
        c.zero_when_cp_zero = false;
    }

    const bool has_k = c.k.n > 0 || c.k.total == 0;
    // The split form pays for splitting both operands (each read twice, S BF16
    // planes written) and pads M and N to 128-row tiles.  When M or N is at most
    // kSplitMinMN (GEMV-shaped products) the FP64 kernels are faster as well as
    // exact to FP64, so they run instead and the split report shows 0 slices.
    constexpr int64_t kSplitMinMN = 4;
    if (opt.precision == EG_PRECISION_SPLIT_BF16 && c.k.total > 0 && c.m.total > kSplitMinMN &&
        c.n.total > kSplitMinMN) {
        eg_split_report rep{};
        st = launch_split_contract(c, opt.slices, stream, &rep);
        if (st == EG_SUCCESS) set_split_report(rep);
        return st;
    }
    set_split_report(eg_split_report{0, 0, 0, 0.0});
    if (!has_k) return launch_elementwise(c, stream);
    if (c.batch.n == 0 && c.m.n == 0 && c.n.n == 0) return launch_dot(c, stream);
    if (c.m.n == 0 || c.n.n == 0) return launch_gemv(c, stream);
    if (f64_tensor_pays(c)) {
        st = launch_f64_tensor(c, stream);
        if (st != EG_ERROR_NOT_SUPPORTED) return st;
    }
    return launch_contract_f64(c, stream);
}

// Validates, classifies and lowers one item of a batch; gemm_shaped tells
// whether it can join a grouped launch (summed modes, an output with more
// than one position, no repeated output index).  What `pattern` knows of the labels is found
// for the first item and used for the others, which have the same ones.
eg_status lower_for_group(double cp, const int32_t *Cl, const eg_tensor *C, double ab, const int32_t *Al,
                          const eg_tensor *A, const int32_t *Bl, const eg_tensor *B, const eg_options &opt,
                          Contraction &out, int32_t *alg_out, bool &gemm_shaped, ListPattern &pattern) {
    eg_status st;
    if ((st = check_tensor(C, Cl, "C")) != EG_SUCCESS) return st;
    if ((st = check_tensor(A, Al, "A")) != EG_SUCCESS) return st;
    if ((st = check_tensor(B, Bl, "B")) != EG_SUCCESS) return st;
    if (pattern.ranks[0] != C->rank || pattern.ranks[1] != A->rank || pattern.ranks[2] != B->rank) {
        pattern.analysis = std::make_shared<detail::Analysis>(labels_of(Cl, C->rank), labels_of(Al, A->rank),
                                                              labels_of(Bl, B->rank));
        pattern.algorithm = (int32_t)classify_labels(*pattern.analysis, opt.semantics);
        pattern.ranks[0] = C->rank;
        pattern.ranks[1] = A->rank;
        pattern.ranks[2] = B->rank;
    }
    const Algorithm alg = choose(*pattern.analysis, (Algorithm)pattern.algorithm, opt, C, A, B);
    if (alg_out) *alg_out = (int32_t)alg;
    Lowered low;
    if ((st = lower(Cl, C, Al, A, Bl, B, opt.semantics, low)) != EG_SUCCESS) return st;
    out = low.c;
    out.cp = cp;
    out.ab = ab;
    out.zero_when_cp_zero = !(opt.semantics == EG_SEMANTICS_CPP && (alg == Algorithm::DOT || alg == Algorithm::GER));
    bool c_repeats = false;
    for (int i = 0; i < C->rank; i++)
        for (int j = i + 1; j < C->rank; j++) c_repeats |= Cl[i] == Cl[j];
    gemm_shaped = !low.empty_c && !c_repeats && out.k.n > 0 && out.k.total > 0 &&
                  (out.m.n > 0 || out.n.n > 0 || out.batch.n > 0);
    return EG_SUCCESS;
}

eg_status build_permute_desc(double cp, const int32_t *Cl, const eg_tensor *C, double ap, const int32_t *Al,
                             const eg_tensor *A, PermuteDesc &p) {
    eg_status st;
    if ((st = check_tensor(C, Cl, "C")) != EG_SUCCESS) return st;
    if ((st = check_tensor(A, Al, "A")) != EG_SUCCESS) return st;
    if (C->rank != A->rank) return fail(EG_ERROR_RANK, "permute: C and A ranks differ");
    p = PermuteDesc{};
    p.rank = C->rank;
    p.A = A->data;
    p.C = C->data;
    p.cp = cp;
    p.ap = ap;
    for (int d = 0; d < C->rank; d++) {
        int where = -1, count = 0;
        for (int j = 0; j < A->rank; j++)
            if (Al[j] == Cl[d]) {
                where = j;
                count++;
            }
        if (count != 1) return fail(EG_ERROR_INVALID_ARGUMENT, "permute: every C index must occur exactly once in A");
        if (C->extent[d] < A->extent[where])
            return fail(EG_ERROR_DIMENSION, "permute: dimension " + std::to_string(d) +
                                                " of the output tensor is smaller than the input tensor");
        p.ext[d] = A->extent[where];
        p.sA[d] = A->stride[where];
        p.sC[d] = C->stride[d];
    }
    for (int j = 0; j < A->rank; j++) {
        int count = 0;
        for (int d = 0; d < C->rank; d++) count += (Cl[d] == Al[j]);
        if (count != 1) return fail(EG_ERROR_INVALID_ARGUMENT, "permute: every A index must occur exactly once in C");
    }
    return EG_SUCCESS;
}

eg_status permute_impl(double cp, const int32_t *Cl, const eg_tensor *C, double ap, const int32_t *Al,
                       const eg_tensor *A, cudaStream_t stream) {
    PermuteDesc p;
    const eg_status st = build_permute_desc(cp, Cl, C, ap, Al, A, p);
    if (st != EG_SUCCESS) return st;
    return launch_permute(p, stream);
}

} // namespace eg

extern "C" {

void eg_options_default(eg_options *opt) {
    if (!opt) return;
    opt->precision = EG_PRECISION_FP64;
    opt->slices = 0;
    opt->tolerance = 1e-10;
    opt->semantics = EG_SEMANTICS_CPP;
    opt->only_generic = 0;
}

eg_status eg_einsum(double C_prefactor, const int32_t *C_labels, const eg_tensor *C, double AB_prefactor,
                    const int32_t *A_labels, const eg_tensor *A, const int32_t *B_labels, const eg_tensor *B,
                    const eg_options *opt, void *stream, int32_t *algorithm_choice) {
    eg::set_error("");
    try {
        return eg::einsum_impl(C_prefactor, C_labels, C, AB_prefactor, A_labels, A, B_labels, B, opt,
                               (cudaStream_t)stream, algorithm_choice);
    } catch (const std::exception &e) {
        return eg::fail(EG_ERROR_INVALID_ARGUMENT, e.what());
    } catch (...) {
        return eg::fail(EG_ERROR_INVALID_ARGUMENT, "unknown exception");
    }
}

eg_status eg_classify(int32_t C_rank, const int32_t *C_labels, int32_t A_rank, const int32_t *A_labels, int32_t B_rank,
                      const int32_t *B_labels, int32_t semantics, int32_t *algorithm_choice) {
    eg::set_error("");
    if (!algorithm_choice) return eg::fail(EG_ERROR_INVALID_ARGUMENT, "algorithm_choice is NULL");
    for (int32_t r : {C_rank, A_rank, B_rank})
        if (r < 0 || r > EG_MAX_RANK) return eg::fail(EG_ERROR_RANK, "rank out of range");
    if ((C_rank && !C_labels) || (A_rank && !A_labels) || (B_rank && !B_labels))
        return eg::fail(EG_ERROR_INVALID_ARGUMENT, "labels are NULL");
    const eg::detail::Analysis an(eg::labels_of(C_labels, C_rank), eg::labels_of(A_labels, A_rank),
                                  eg::labels_of(B_labels, B_rank));
    *algorithm_choice = (int32_t)eg::classify_labels(an, semantics);
    return EG_SUCCESS;
}

eg_status eg_permute(double C_prefactor, const int32_t *C_labels, const eg_tensor *C, double A_prefactor,
                     const int32_t *A_labels, const eg_tensor *A, void *stream) {
    eg::set_error("");
    try {
        return eg::permute_impl(C_prefactor, C_labels, C, A_prefactor, A_labels, A, (cudaStream_t)stream);
    } catch (...) {
        return eg::fail(EG_ERROR_INVALID_ARGUMENT, "exception in eg_permute");
    }
}

eg_status eg_einsum_batched(double C_prefactor, const int32_t *C_labels, const eg_tensor *C_list, double AB_prefactor,
                            const int32_t *A_labels, const eg_tensor *A_list, const int32_t *B_labels,
                            const eg_tensor *B_list, int64_t count, const eg_options *opt, void *stream,
                            int32_t *algorithm_choice);

eg_status eg_last_split_report(eg_split_report *out) {
    if (!out) return eg::fail(EG_ERROR_INVALID_ARGUMENT, "out is NULL");
    *out = eg::g_split_report;
    return EG_SUCCESS;
}

eg_status eg_device_alloc(size_t bytes, void **ptr) {
    eg::set_error("");
    if (!ptr) return eg::fail(EG_ERROR_INVALID_ARGUMENT, "ptr is NULL");
    return eg::tracked_malloc(bytes, ptr);
}

eg_status eg_device_free(void *ptr) {
    eg::set_error("");
    return eg::tracked_free(ptr);
}

eg_status eg_set_memory_budget(size_t bytes) {
    std::lock_guard<std::mutex> lk(eg::g_mem_mutex);
    eg::g_budget = bytes;
    return EG_SUCCESS;
}

eg_status eg_memory_in_use(size_t *bytes) {
    if (!bytes) return eg::fail(EG_ERROR_INVALID_ARGUMENT, "bytes is NULL");
    std::lock_guard<std::mutex> lk(eg::g_mem_mutex);
    *bytes = eg::g_in_use;
    return EG_SUCCESS;
}

eg_status eg_trim_memory(void) {
    eg::set_error("");
    try {
        eg::RelaxedCapture relaxed;
        eg::trim_scratch();
        eg::drop_cached_plans();
        return EG_SUCCESS;
    } catch (const std::exception &e) {
        return eg::fail(EG_ERROR_OUT_OF_MEMORY, e.what());
    }
}

eg_status eg_copy_to_device(void *dst, const void *src, size_t bytes, void *stream) {
    EG_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, (cudaStream_t)stream));
    return EG_SUCCESS;
}

eg_status eg_copy_to_host(void *dst, const void *src, size_t bytes, void *stream) {
    EG_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    return EG_SUCCESS;
}

eg_status eg_stream_synchronize(void *stream) {
    EG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return EG_SUCCESS;
}

eg_status eg_stream_status(void *stream, int32_t *device_code) {
    eg::set_error("");
    int *w = nullptr;
    eg_status st = eg::status_word((cudaStream_t)stream, &w);
    if (st != EG_SUCCESS) return st;
    EG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    int code = 0;
    EG_CUDA(cudaMemcpy(&code, w, sizeof(int), cudaMemcpyDeviceToHost));
    if (code) EG_CUDA(cudaMemset(w, 0, sizeof(int)));
    if (device_code) *device_code = code;
    if (code) return eg::fail(EG_ERROR_TIMEOUT, "a bounded device wait gave up (code " + std::to_string(code) + ")");
    return EG_SUCCESS;
}

const char *eg_last_error(void) { return eg::g_last_error.c_str(); }

const char *eg_status_string(eg_status s) {
    switch (s) {
    case EG_SUCCESS: return "success";
    case EG_ERROR_INVALID_ARGUMENT: return "invalid argument";
    case EG_ERROR_RANK: return "rank error";
    case EG_ERROR_DIMENSION: return "dimension error";
    case EG_ERROR_NOT_SUPPORTED: return "not supported";
    case EG_ERROR_CUDA: return "CUDA error";
    case EG_ERROR_OUT_OF_MEMORY: return "out of memory";
    case EG_ERROR_TIMEOUT: return "device wait timed out";
    case EG_ERROR_PRECISION: return "precision target not reachable";
    }
    return "unknown status";
}

const char *eg_version(void) { return "einsums_gb300 0.1.0 (sm_103a)"; }

} // extern "C"
