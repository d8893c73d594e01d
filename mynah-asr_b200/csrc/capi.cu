// extern "C" boundary (include/mynah_b200.h): plain pointers and sizes in, host
// buffers out; resolves the reference's tensor names and drives the device path.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <memory>

#include "hostcopy.h"
#include "model.h"

using namespace mb;

namespace mb { long long launch_count(bool reset); }

// A model handle = the immutable weights + a small pool of execution contexts. Context 0 is `m` itself; further
// contexts are shallow copies of it made on demand (same device pointers to the weights, their own CUDA stream,
// workspace arena, status word and profiling state), so calls from several host threads run side by side on the
// same weights — the counterpart of the reference's per-thread cuBLAS handle / stream / buffers over a shared
// weight cache (src/cuda_gemm.cu:50-60,92-130).
struct mynah_b200_model {
    CopyUser copies;
    Model m;
    std::vector<std::unique_ptr<Model>> extra;      // contexts 1..
    std::vector<char> busy{0};                      // per context
    std::mutex pool_mu;
    std::condition_variable pool_cv;
    int max_ctx = 4;
    int device = 0;                                 // the GPU the model lives on
    Model &ctx(int i) { return i == 0 ? m : *extra[(size_t)i - 1]; }
    int n_ctx() const { return 1 + (int)extra.size(); }
};

namespace {
// Takes a free context for the duration of a call (lowest index first, so a single-threaded caller always runs on
// context 0); creates one while fewer than max_ctx exist, else waits. want >= 0: that context and no other (a
// stream group's caches and captured graph belong to the context that opened it).
class Lease {
public:
    explicit Lease(mynah_b200_model *h, int want = -1) : h_(h) {
        cudaSetDevice(h->device);                    // a fresh host thread starts on device 0
        std::unique_lock<std::mutex> lk(h->pool_mu);
        for (;;) {
            if (want >= 0) {
                if (want < h->n_ctx() && !h->busy[(size_t)want]) { idx_ = want; break; }
            } else {
                for (int i = 0; i < h->n_ctx(); i++) if (!h->busy[(size_t)i]) { idx_ = i; break; }
                if (idx_ >= 0) break;
                if (h->n_ctx() < h->max_ctx && h->m.finalized) {
                    if (Model *c = clone_context(h->m)) {
                        h->extra.emplace_back(c);
                        h->busy.push_back(0);
                        idx_ = h->n_ctx() - 1;
                        break;
                    }
                }
            }
            h->pool_cv.wait(lk);
        }
        h->busy[(size_t)idx_] = 1;
    }
    ~Lease() {
        if (!idle_) model().settle();
        { std::lock_guard<std::mutex> lk(h_->pool_mu); h_->busy[(size_t)idx_] = 0; }
        h_->pool_cv.notify_all();
    }
    Model &model() { return h_->ctx(idx_); }
    int index() const { return idx_; }
    // the call's last act was to wait, with success, for everything it issued: no need to ask the streams (3 us)
    void idle() { idle_ = true; }
    Lease(const Lease &) = delete;
    Lease &operator=(const Lease &) = delete;

private:
    static Model *clone_context(const Model &src) {
        Model *c = new Model(src);                   // weights: the same device pointers
        c->owned.clear();                            // ... which only context 0 owns
        c->slabs.clear(); c->use_slabs = false;
        for (int i = 0; i < Model::DEC_LANES; i++) { c->lane[i] = nullptr; c->lane_done[i] = nullptr; }
        c->lane_fork = nullptr;
        c->prof_spans.clear(); c->prof_used = 0; c->prof_on = false;
        c->ws = Arena(); c->host_stage = HostStage();
        c->copy = nullptr; c->copy_ev.clear();
        c->stream = nullptr; c->status = nullptr;
        if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) { cudaGetLastError(); delete c; return nullptr; }
        c->status = (int *)c->dev_alloc(sizeof(int));
        if (!c->status || cudaMemset(c->status, 0, sizeof(int)) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) { delete c; return nullptr; }
        return c;
    }
    mynah_b200_model *h_;
    int idx_ = -1;
    bool idle_ = false;
};

// Runs fn on every context while none of them is in a call.
template <typename F>
void with_all_contexts_idle(mynah_b200_model *h, F fn) {
    std::unique_lock<std::mutex> lk(h->pool_mu);
    h->pool_cv.wait(lk, [&] { for (char b : h->busy) if (b) return false; return true; });
    for (int i = 0; i < h->n_ctx(); i++) fn(h->ctx(i));
}
}  // namespace
// A resident weight and what its products need.
//   block  device [status, 256 B | QMAT_SMALL out | QMAT_SMALL x | temporaries of that x]: a small call moves its rows in with
//          one copy and the result with the status word out with one copy, through a pinned twin
// Anything larger comes from the workspaces that all handles of a device share (WorkspacePool). Allocating it per call
// cost 0.48 ms of a 16 us product: the stream-ordered pool gives its memory back at every synchronisation and maps it anew at
// the next allocation; a workspace per handle moves that cost into the first product of each of a model's linears (187 rows
// of [1024 x 4096]: 680 us instead of 309).
// One lock per handle: products of one weight share the block and run one after the other on the handle's stream.
struct mynah_b200_qmat {
    CopyUser copies;
    QWeight w;
    std::vector<void *> owned;
    cudaStream_t stream = nullptr;
    int *status = nullptr;               // = the first word of the block
    int device = 0;
    uint64_t id = 0;                     // never used again, unlike an address or a stream
    mutable std::mutex mu;
    mutable uint8_t *host = nullptr;     // the block's pinned twin, once a graph names it; until then a call borrows one
    // A small call repeated with the same rows and flags is one graph (copy in, kernels, copy out) instead of four or five
    // pieces: 29.5 us against 34.4 for one row of [4096 x 1024], 51 against 57 for 32 of [1024 x 1024]. Recording takes 70 us, so
    // it waits for the second such call. Four of them, for a program that alternates between a few row counts; a fifth takes the
    // oldest one's place and runs in pieces until it comes again.
    struct Graph { int T = 0, flags = 0, uses = 0, launches = 0; cudaGraphExec_t exec = nullptr; };
    mutable Graph graphs[4];
    mutable int graph_next = 0;
};
// Rows or results up to QMAT_SMALL bytes go through the block. With 32 rows of [1024 x 1024], 128 KB each way, a product takes
// 51 us that way and 65 by copies of their own from pageable memory. It would still take 101 against 118 us at 512 KB: the
// line is what every handle of a model holds for it, three times this on the device.
static constexpr size_t QMAT_HEAD = 256, QMAT_SMALL = 128 << 10;
static constexpr size_t QMAT_TEMP_AT = QMAT_HEAD + 2 * QMAT_SMALL, QMAT_TEMP = QMAT_SMALL + 512;   // two fp16 planes of x, aligned
static constexpr size_t QMAT_PINNED = QMAT_TEMP_AT, QMAT_BLOCK = QMAT_TEMP_AT + QMAT_TEMP;
static constexpr size_t QMAT_KEEP = 64 << 20;
struct mynah_b200_batch {
    int batch = 0;
    std::vector<float *> audio;          // device
    std::vector<size_t> n_samples;
    std::vector<std::vector<int>> tokens, frames;
    std::vector<int> prompt_ids;         // prompt-conditioned encoders: one id per utterance (empty = 0 for all)
    std::vector<int> aed_prompt;         // decoder 2 (AED): the prompt every utterance starts from,
    int aed_eos = -1, aed_delta = 0;     // the end-of-sequence id and the generation allowance beyond T
};

struct mynah_b200_stream_group {
    mynah_b200_model *model = nullptr;
    int ctx = 0;                         // the execution context the group lives on
    mb::StreamState st;
};

namespace mb {
void set_load_seconds(mynah_b200_model *h, double seconds) { if (h) h->m.load_seconds = seconds; }
QmatView qmat_view(const void *handle) {
    const mynah_b200_qmat *q = static_cast<const mynah_b200_qmat *>(handle);
    return QmatView{&q->w, q->stream};
}
}  // namespace mb

namespace {
// Pinned twins of the handles' blocks. Pinning costs more than a product, so up to POOL_MAX free ones (8 MB) stay, for the
// next call that borrows one and beyond the handles.
class PinnedPool {
public:
    uint8_t *take() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (!free_.empty()) { uint8_t *p = free_.back(); free_.pop_back(); return p; }
        }
        void *p = nullptr;
        if (cudaHostAlloc(&p, QMAT_PINNED, cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        return (uint8_t *)p;
    }
    void give(uint8_t *p) {
        if (!p) return;
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (free_.size() < POOL_MAX) { free_.push_back(p); return; }
        }
        cudaFreeHost(p);
    }

private:
    static constexpr size_t POOL_MAX = 32;
    std::mutex mu_;
    std::vector<uint8_t *> free_;
};
PinnedPool &pinned_pool() { static PinnedPool *p = new PinnedPool(); return *p; }   // alive until the process ends

// The pinned twin for one call: the handle's own, or one that goes back when the call ends (it has waited for its stream by
// then) unless a graph has come to name it.
class PinnedTwin {
public:
    explicit PinnedTwin(const mynah_b200_qmat *q) : q_(q), p_(q->host ? q->host : pinned_pool().take()) {}
    ~PinnedTwin() { if (p_ != q_->host) pinned_pool().give(p_); }
    uint8_t *get() const { return p_; }
    void keep() { q_->host = p_; }
    PinnedTwin(const PinnedTwin &) = delete;
    PinnedTwin &operator=(const PinnedTwin &) = delete;

private:
    const mynah_b200_qmat *q_;
    uint8_t *p_;
};

// Device workspaces of the products, shared by the handles of a device. A call takes a block for as long as it issues work
// and gives it back with an event behind that work; whoever takes it next waits for the event on its own stream (the same
// handle need not: its products share a stream). A block whose work has finished goes first, then a fresh one while fewer than
// KEEP_BLOCKS are free, so that products of several handles still overlap. Free blocks are at most KEEP_BLOCKS per device, of
// at most QMAT_KEEP bytes each, and all go when the device's last handle does.
struct Workspace { uint8_t *p = nullptr; size_t cap = 0; int device = 0; uint64_t user = 0; cudaEvent_t done = nullptr; };
class WorkspacePool {
public:
    int handle_made() { const int dev = current(); std::lock_guard<std::mutex> lk(mu_); handles_[dev]++; return dev; }
    void handle_gone(int dev) {
        std::vector<Workspace> drop;
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (--handles_[dev] > 0) return;
            for (size_t i = 0; i < free_.size();)
                if (free_[i].device == dev) { drop.push_back(free_[i]); free_.erase(free_.begin() + i); } else i++;
        }
        for (Workspace &w : drop) destroy(w);
    }
    // Workspace::p is null on failure
    Workspace take(size_t bytes, uint64_t user, cudaStream_t st) {
        RelaxedCapture relaxed;
        Workspace w;
        w.device = current();
        {
            std::lock_guard<std::mutex> lk(mu_);
            int best = -1, waits = -1, here = 0;
            for (int i = 0; i < (int)free_.size(); i++) {
                const Workspace &f = free_[(size_t)i];
                if (f.device != w.device) continue;
                here++;
                if (f.cap < bytes) continue;
                int &pick = f.user == user || cudaEventQuery(f.done) == cudaSuccess ? best : waits;
                if (pick < 0 || f.cap < free_[(size_t)pick].cap) pick = i;
            }
            cudaGetLastError();                                  // "not ready" is noted as an error
            if (best < 0 && here >= KEEP_BLOCKS) best = waits;
            if (best >= 0) { w = free_[(size_t)best]; free_.erase(free_.begin() + best); }
        }
        if (w.p) {
            if (w.user != user && cudaStreamWaitEvent(st, w.done, 0) != cudaSuccess) { cudaGetLastError(); cudaEventSynchronize(w.done); }
            return w;
        }
        w.cap = 1 << 20;
        while (w.cap < bytes) w.cap <<= 1;
        if (cudaEventCreateWithFlags(&w.done, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); return Workspace(); }
        if (cudaMalloc((void **)&w.p, w.cap) != cudaSuccess) { cudaGetLastError(); cudaEventDestroy(w.done); return Workspace(); }
        return w;
    }
    void give(Workspace w, uint64_t user, cudaStream_t st) {
        w.user = user;
        if (cudaEventRecord(w.done, st) != cudaSuccess) { cudaGetLastError(); cudaStreamSynchronize(st); destroy(w); return; }
        {
            std::lock_guard<std::mutex> lk(mu_);
            free_.push_back(w);
            int here = 0;
            size_t least = free_.size() - 1;
            for (size_t i = 0; i < free_.size(); i++)
                if (free_[i].device == w.device) { here++; if (free_[i].cap < free_[least].cap) least = i; }
            if (here <= KEEP_BLOCKS) return;
            w = free_[least];
            free_.erase(free_.begin() + (long)least);
        }
        destroy(w);
    }

private:
    static constexpr int KEEP_BLOCKS = 4;
    static int current() { int d = 0; if (cudaGetDevice(&d) != cudaSuccess) cudaGetLastError(); return d; }
    static void destroy(Workspace &w) { RelaxedCapture relaxed; cudaEventSynchronize(w.done); cudaEventDestroy(w.done); cudaFree(w.p); cudaGetLastError(); }
    std::mutex mu_;
    std::vector<Workspace> free_;
    std::map<int, int> handles_;
};
WorkspacePool &workspace_pool() { static WorkspacePool *p = new WorkspacePool(); return *p; }   // alive until the process ends

// `bytes` of device workspace for what a call issues on a handle whose lock is held: a shared block, or (above QMAT_KEEP) a
// stream-ordered allocation that ends with the call.
class QmatScratch {
public:
    QmatScratch(const mynah_b200_qmat *q, size_t bytes) : q_(q) {
        if (bytes == 0) return;
        if (bytes > QMAT_KEEP) {
            if (cudaMallocAsync(&own_, bytes, q->stream) != cudaSuccess) { cudaGetLastError(); own_ = nullptr; }
        } else {
            ws_ = workspace_pool().take(bytes, q->id, q->stream);
        }
    }
    ~QmatScratch() {
        if (own_) cudaFreeAsync(own_, q_->stream);
        if (ws_.p) workspace_pool().give(ws_, q_->id, q_->stream);
    }
    uint8_t *get() const { return own_ ? (uint8_t *)own_ : ws_.p; }
    QmatScratch(const QmatScratch &) = delete;
    QmatScratch &operator=(const QmatScratch &) = delete;

private:
    const mynah_b200_qmat *q_;
    Workspace ws_;
    void *own_ = nullptr;
};
}  // namespace

static int internal_fmt(int fmt) {
    switch (fmt) {
    case MYNAH_B200_F32: return FMT_F32;
    case MYNAH_B200_MYNAH_Q8: return FMT_MYNAH_Q8;
    case MYNAH_B200_MYNAH_Q4: return FMT_MYNAH_Q4;
    case MYNAH_B200_GGML_Q4_0: return FMT_GGML_Q4_0;
    case MYNAH_B200_GGML_Q8_0: return FMT_GGML_Q8_0;
    case MYNAH_B200_GGML_Q4_K: return FMT_GGML_Q4_K;
    case MYNAH_B200_GGML_Q6_K: return FMT_GGML_Q6_K;
    default: return -1;
    }
}

extern "C" {

const char *mynah_b200_last_error(void) { return mb::last_error(); }

int mynah_b200_available(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0) { cudaGetLastError(); return 0; }
    int dev = 0, major = 0, minor = 0;
    cudaGetDevice(&dev);                               // two attributes: the whole property block takes milliseconds to fill
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev) != cudaSuccess) { cudaGetLastError(); return 0; }
    return major == 10 && minor == 0 ? 1 : 0;          // the library holds sm_100a code only
}

int mynah_b200_select_device(int index) {
    if (index < 0) {
        const char *e = getenv("MYNAH_B200_DEVICE");
        if (!e) e = getenv("LOCAL_RANK");
        index = e ? atoi(e) : 0;
    }
    int n = 0;
    MB_CUDA(cudaGetDeviceCount(&n));
    if (index >= n) { set_error("device %d requested, %d present", index, n); return -1; }
    MB_CUDA(cudaSetDevice(index));
    return index;
}

long long mynah_b200_launch_count(int reset) { return mb::launch_count(reset != 0); }

void mynah_b200_config_default(mynah_b200_config *c) {
    memset(c, 0, sizeof(*c));
    c->n_mels = 128; c->n_fft = 512; c->win_length = 400; c->hop_length = 160;
    c->preemphasis = 0.97; c->log_zero_guard = 5.9604644775390625e-8;
    c->normalize_per_feature = 1; c->causal = -1; c->xscaling = 0;
    c->left_ctx = -1; c->right_ctx = -1; c->blank_id = 0; c->max_symbols = 10;
    c->n_durations = 0; c->strict = 1; c->attn_impl = 0; c->aed_heads = 8; c->a8 = 0;
}

// ------------------------------------------------------------------- model
mynah_b200_model *mynah_b200_model_new(const mynah_b200_config *cfg) {
    if (!mynah_b200_available()) { set_error("no sm_100 CUDA device available"); return nullptr; }
    mynah_b200_model *h = new mynah_b200_model();
    if (cfg) h->m.cfg = *cfg; else mynah_b200_config_default(&h->m.cfg);
    cudaGetDevice(&h->device);
    if (const char *e = getenv("MYNAH_B200_CONTEXTS")) { const int n = atoi(e); if (n >= 1 && n <= 64) h->max_ctx = n; }
    if (cudaStreamCreateWithFlags(&h->m.stream, cudaStreamNonBlocking) != cudaSuccess) {
        set_error("cudaStreamCreate failed"); delete h; return nullptr;
    }
    h->m.status = (int *)h->m.dev_alloc(sizeof(int));
    if (!h->m.status) { delete h; return nullptr; }
    h->m.use_slabs = true;
    cudaMemset(h->m.status, 0, sizeof(int));
    cudaDeviceSynchronize();
    return h;
}

int mynah_b200_model_add_tensor(mynah_b200_model *h, const char *name, int fmt, const int64_t *shape, int rank,
                                const void *data) {
    if (!h || !name || !data || rank <= 0 || rank > 8) { set_error("add_tensor: bad argument"); return -1; }
    if (h->m.finalized) { set_error("add_tensor after finalize"); return -1; }
    const int f = internal_fmt(fmt);
    if (f < 0) { set_error("add_tensor '%s': unknown format %d", name, fmt); return -1; }
    HostTensor t;
    t.fmt = f; t.data = data; t.shape.assign(shape, shape + rank);
    h->m.host[name] = t;
    return 0;
}

int mynah_b200_model_set_mel(mynah_b200_model *h, const float *mel_fb, const float *window) {
    if (!h || !mel_fb || !window) { set_error("set_mel: bad argument"); return -1; }
    Model &m = h->m;
    const int nb = m.cfg.n_fft / 2 + 1, nm = m.cfg.n_mels, nf = m.cfg.n_fft;
    m.mel_fb = m.upload_f32(mel_fb, (size_t)nb * nm);
    // non-zero bin range per filter, as mel_ranges does (src/features.c:50-61)
    std::vector<int> lo(nm), hi(nm);
    for (int k = 0; k < nm; k++) {
        int a = nb, z = 0;
        for (int b = 0; b < nb; b++) if (mel_fb[(size_t)b * nm + k] != 0.0f) { if (b < a) a = b; z = b + 1; }
        lo[k] = a; hi[k] = z;
    }
    std::vector<double> win(nf, 0.0), tw(nf);
    const int off = (nf - m.cfg.win_length) / 2;
    for (int i = 0; i < m.cfg.win_length; i++) win[off + i] = (double)window[i];
    for (int j = 0; j < nf / 2; j++) { const double a = -2.0 * M_PI * j / nf; tw[2 * j] = cos(a); tw[2 * j + 1] = sin(a); }
    m.mel_lo = (int *)m.dev_alloc(nm * sizeof(int));
    m.mel_hi = (int *)m.dev_alloc(nm * sizeof(int));
    m.mel_win = (double *)m.dev_alloc(nf * sizeof(double));
    m.mel_tw = (double *)m.dev_alloc(nf * sizeof(double));
    if (!m.mel_fb || !m.mel_lo || !m.mel_hi || !m.mel_win || !m.mel_tw) return -1;
    MB_CUDA(cudaMemcpy(m.mel_lo, lo.data(), nm * sizeof(int), cudaMemcpyHostToDevice));
    MB_CUDA(cudaMemcpy(m.mel_hi, hi.data(), nm * sizeof(int), cudaMemcpyHostToDevice));
    MB_CUDA(cudaMemcpy(m.mel_win, win.data(), nf * sizeof(double), cudaMemcpyHostToDevice));
    MB_CUDA(cudaMemcpy(m.mel_tw, tw.data(), nf * sizeof(double), cudaMemcpyHostToDevice));
    MB_CUDA(cudaDeviceSynchronize());     // these went through the legacy stream; the model's stream does not wait on it
    m.has_mel = true;
    return 0;
}

}  // extern "C"

// ---- name resolution helpers
static const HostTensor *find(Model &m, const std::string &name) {
    auto it = m.host.find(name);
    return it == m.host.end() ? nullptr : &it->second;
}
static const float *f32dev(Model &m, const std::string &name, bool required, int *err) {
    const HostTensor *t = find(m, name);
    if (!t) { if (required) { set_error("missing tensor '%s'", name.c_str()); *err = 1; } return nullptr; }
    if (t->fmt != FMT_F32) { set_error("tensor '%s' must be f32", name.c_str()); *err = 1; return nullptr; }
    float *d = m.upload_f32((const float *)t->data, t->nelem());
    if (!d) *err = 1;
    return d;
}
// a linear [n, k] or [n, k, 1]; bias looked up beside it
static int lin(Model &m, QWeight &w, const std::string &wname, bool planes, bool want_f32, const int *perm = nullptr) {
    const HostTensor *t = find(m, wname);
    if (!t || t->shape.empty() || t->shape[0] <= 0) { set_error("missing tensor '%s'", wname.c_str()); return -1; }
    const int n = (int)t->shape[0], k = (int)(t->nelem() / (size_t)t->shape[0]);
    const HostTensor *ts = find(m, wname + ".scales");     // native quantised checkpoints
    if (m.upload_weight(w, t->fmt, t->data, ts ? (const float *)ts->data : nullptr, n, k, planes, want_f32, perm)) return -1;
    std::string bname = wname;
    const size_t p = bname.rfind(".weight");
    if (p != std::string::npos) bname.replace(p, 7, ".bias");
    int err = 0;
    w.bias = const_cast<float *>(f32dev(m, bname, false, &err));
    return err ? -1 : 0;
}

// q, k and v of a layer read the same rows: their operands (planes, or natively quantised bytes and scales) get one block,
// so that L.qkv is all three as one [3 d, d] weight and q_w, k_w, v_w are parts of it
static int place_qkv(Model &m, EncLayer &L, const std::string &p) {
    const char *names[3] = {"q_proj", "k_proj", "v_proj"};
    const int d = m.d_model;
    const size_t dd = (size_t)d * d;
    bool native8 = true;
    for (const char *nm : names) {
        const HostTensor *t = find(m, p + "self_attn." + nm + ".weight");
        if (!t || t->shape.empty()) { set_error("missing tensor '%sself_attn.%s.weight'", p.c_str(), nm); return -1; }
        if (t->shape[0] != d || t->nelem() != dd) { set_error("'%sself_attn.%s.weight' is not [%d, %d]", p.c_str(), nm, d, d); return -1; }
        native8 = native8 && t->fmt == FMT_MYNAH_Q8;
    }
    QWeight &w = L.qkv;
    w.n = 3 * d; w.k = d;
    w.hi = (__half *)m.dev_alloc(3 * dd * 2); w.lo = (__half *)m.dev_alloc(3 * dd * 2);
    if (!w.hi || !w.lo) return -1;
    if (native8) {
        w.fmt = FMT_MYNAH_Q8;
        w.raw = (uint8_t *)m.dev_alloc(3 * dd + 64); w.scales = (float *)m.dev_alloc(3 * (size_t)d * 4);
        if (!w.raw || !w.scales) return -1;
    }
    QWeight *parts[3] = {&L.q_w, &L.k_w, &L.v_w};
    for (int i = 0; i < 3; i++) {
        parts[i]->hi = w.hi + i * dd; parts[i]->lo = w.lo + i * dd;
        if (native8) { parts[i]->raw = w.raw + i * dd; parts[i]->scales = w.scales + (size_t)i * d; }
    }
    return 0;
}
static int finish_qkv(Model &m, EncLayer &L) {
    const int d = m.d_model;
    const float *b[3] = {L.q_w.bias, L.k_w.bias, L.v_w.bias};
    if (!b[0] && !b[1] && !b[2]) return 0;
    L.qkv.bias = (float *)m.dev_alloc(3 * (size_t)d * 4);
    if (!L.qkv.bias) return -1;
    MB_CUDA(cudaMemsetAsync(L.qkv.bias, 0, 3 * (size_t)d * 4, m.stream));
    for (int i = 0; i < 3; i++)
        if (b[i]) MB_CUDA(cudaMemcpyAsync(L.qkv.bias + (size_t)i * d, b[i], (size_t)d * 4, cudaMemcpyDeviceToDevice, m.stream));
    return 0;
}

// several linears over the same input, stored one below the other: [sum n, k] with the biases concatenated
// (block formats keep whole rows of blocks, so the stored bytes concatenate as they are)
static int lin_cat(Model &m, QWeight &w, const float **bias, const std::vector<std::string> &prefixes) {
    std::vector<uint8_t> bytes;
    std::vector<float> b;
    int fmt = -1, k = 0, n = 0;
    for (const std::string &pre : prefixes) {
        const HostTensor *t = find(m, pre + ".weight"), *tb = find(m, pre + ".bias");
        if (!t || t->shape.size() != 2 || !tb || tb->fmt != FMT_F32) { set_error("missing tensor '%s.weight' or its bias", pre.c_str()); return -1; }
        if (t->fmt == FMT_MYNAH_Q8 || t->fmt == FMT_MYNAH_Q4) { set_error("'%s': natively quantised AED weights are not supported", pre.c_str()); return -1; }
        if (fmt < 0) { fmt = t->fmt; k = (int)t->shape[1]; }
        if (t->fmt != fmt || (int)t->shape[1] != k) { set_error("'%s': projections of one attention differ in format or width", pre.c_str()); return -1; }
        const size_t nb = format_bytes(fmt, (int)t->shape[0], k);
        bytes.insert(bytes.end(), (const uint8_t *)t->data, (const uint8_t *)t->data + nb);
        b.insert(b.end(), (const float *)tb->data, (const float *)tb->data + t->shape[0]);
        n += (int)t->shape[0];
    }
    if (m.upload_weight(w, fmt, bytes.data(), nullptr, n, k, true, false)) return -1;
    *bias = m.upload_f32(b.data(), b.size());
    return *bias ? 0 : -1;
}

extern "C" {

int mynah_b200_model_finalize(mynah_b200_model *h) {
    if (!h) { set_error("finalize: null model"); return -1; }
    Model &m = h->m;
    if (m.finalized) return 0;
    const auto t_load0 = std::chrono::steady_clock::now();
    int err = 0;
    const std::string ss = "encoder.subsampling.";
    std::string cin, dwn[2], pwn[2];
    int causal_naming;
    if (find(m, ss + "conv_in.weight")) {           // Nemotron naming (src/subsampling.c:16-35)
        causal_naming = 1; cin = ss + "conv_in";
        for (int i = 0; i < 2; i++) { dwn[i] = ss + "layers." + std::to_string(i) + ".depthwise_conv"; pwn[i] = ss + "layers." + std::to_string(i) + ".pointwise_conv"; }
    } else {                                        // Parakeet naming (src/subsampling.c:36-52)
        causal_naming = 0; cin = ss + "layers.0";
        dwn[0] = ss + "layers.2"; dwn[1] = ss + "layers.5"; pwn[0] = ss + "layers.3"; pwn[1] = ss + "layers.6";
    }
    m.causal = m.cfg.causal >= 0 ? m.cfg.causal : causal_naming;
    const HostTensor *tc = find(m, cin + ".weight"), *tl = find(m, ss + "linear.weight");
    if (!tc || !tl) { set_error("missing subsampling tensors"); return -1; }
    m.channels = (int)tc->shape[0];
    m.d_model = (int)tl->shape[0];
    m.conv_in_w = f32dev(m, cin + ".weight", true, &err);
    m.conv_in_b = f32dev(m, cin + ".bias", true, &err);
    for (int i = 0; i < 2 && !err; i++) {
        m.dw_w[i] = f32dev(m, dwn[i] + ".weight", true, &err);
        m.dw_b[i] = f32dev(m, dwn[i] + ".bias", true, &err);
        if (lin(m, m.pw[i], pwn[i] + ".weight", true, false)) return -1;
        if (!m.pw[i].bias) { set_error("missing '%s.bias'", pwn[i].c_str()); return -1; }
    }
    if (err) return -1;
    {   // channel-major flatten c*F'+f  ->  f*C+c (see subsampling.cu)
        const int CF = (int)tl->shape[1], C = m.channels, F3 = CF / C;
        int f = m.cfg.n_mels;
        for (int i = 0; i < 3; i++) f = Model::sub_len(f, m.causal);
        if (f != F3) { set_error("subsampling linear expects %d freq bins, n_mels=%d gives %d", F3, m.cfg.n_mels, f); return -1; }
        std::vector<int> perm(CF);
        for (int ff = 0; ff < F3; ff++) for (int c = 0; c < C; c++) perm[ff * C + c] = c * F3 + ff;
        if (lin(m, m.ss_lin, ss + "linear.weight", true, false, perm.data())) return -1;
        if (!m.ss_lin.bias) { set_error("missing subsampling linear bias"); return -1; }
    }
    const HostTensor *bu = find(m, "encoder.layers.0.self_attn.bias_u");
    const HostTensor *dw = find(m, "encoder.layers.0.conv.depthwise_conv.weight");
    if (!bu || !dw) { set_error("missing encoder.layers.0 tensors"); return -1; }
    m.n_heads = (int)bu->shape[0]; m.d_head = (int)bu->shape[1]; m.conv_k = (int)dw->shape[2];
    if (m.cfg.xscaling) m.xscale = sqrtf((float)m.d_model);
    int nl = 0;
    while (find(m, "encoder.layers." + std::to_string(nl) + ".norm_out.weight")) nl++;
    if (nl == 0) { set_error("no encoder layers found"); return -1; }
    m.n_layers = nl;
    m.layers.resize(nl);
    const bool bn = find(m, "encoder.layers.0.conv.norm.running_mean") != nullptr;
    // the layers' rel-pos projections sit one below the other ([layers d, d]): one contraction makes the keys of all layers
    const size_t dd = (size_t)m.d_model * m.d_model;
    __half *relk_hi = (__half *)m.dev_alloc(nl * dd * 2), *relk_lo = (__half *)m.dev_alloc(nl * dd * 2);
    if (!relk_hi || !relk_lo) return -1;
    for (int li = 0; li < nl; li++) {
        EncLayer &L = m.layers[li];
        const std::string p = "encoder.layers." + std::to_string(li) + ".";
        L.ln_ff1_w = f32dev(m, p + "norm_feed_forward1.weight", true, &err); L.ln_ff1_b = f32dev(m, p + "norm_feed_forward1.bias", true, &err);
        L.ln_att_w = f32dev(m, p + "norm_self_att.weight", true, &err); L.ln_att_b = f32dev(m, p + "norm_self_att.bias", true, &err);
        L.ln_conv_w = f32dev(m, p + "norm_conv.weight", true, &err); L.ln_conv_b = f32dev(m, p + "norm_conv.bias", true, &err);
        L.ln_ff2_w = f32dev(m, p + "norm_feed_forward2.weight", true, &err); L.ln_ff2_b = f32dev(m, p + "norm_feed_forward2.bias", true, &err);
        L.ln_out_w = f32dev(m, p + "norm_out.weight", true, &err); L.ln_out_b = f32dev(m, p + "norm_out.bias", true, &err);
        L.bias_u = f32dev(m, p + "self_attn.bias_u", true, &err); L.bias_v = f32dev(m, p + "self_attn.bias_v", true, &err);
        L.dw_w = f32dev(m, p + "conv.depthwise_conv.weight", true, &err);
        L.dw_b = f32dev(m, p + "conv.depthwise_conv.bias", false, &err);
        L.cnorm_w = f32dev(m, p + "conv.norm.weight", true, &err); L.cnorm_b = f32dev(m, p + "conv.norm.bias", true, &err);
        L.cnorm_scale = L.cnorm_shift = nullptr;
        if (err) return -1;
        if (bn) {   // fold BatchNorm running stats (src/encoder.c:149-170)
            const HostTensor *mu = find(m, p + "conv.norm.running_mean"), *var = find(m, p + "conv.norm.running_var");
            const HostTensor *gw = find(m, p + "conv.norm.weight"), *gb = find(m, p + "conv.norm.bias");
            if (!mu || !var) { set_error("missing BatchNorm running stats at layer %d", li); return -1; }
            std::vector<float> sc(m.d_model), sh(m.d_model);
            for (int i = 0; i < m.d_model; i++) {
                sc[i] = (float)((double)((const float *)gw->data)[i] / sqrt((double)((const float *)var->data)[i] + 1e-5));
                sh[i] = ((const float *)gb->data)[i] - ((const float *)mu->data)[i] * sc[i];
            }
            L.cnorm_scale = m.upload_f32(sc.data(), m.d_model);
            L.cnorm_shift = m.upload_f32(sh.data(), m.d_model);
            if (!L.cnorm_scale || !L.cnorm_shift) return -1;
        }
        L.relk.hi = relk_hi + li * dd; L.relk.lo = relk_lo + li * dd;
        if (place_qkv(m, L, p)) return -1;
        if (lin(m, L.ff1_w1, p + "feed_forward1.linear1.weight", true, false) || lin(m, L.ff1_w2, p + "feed_forward1.linear2.weight", true, false) ||
            lin(m, L.ff2_w1, p + "feed_forward2.linear1.weight", true, false) || lin(m, L.ff2_w2, p + "feed_forward2.linear2.weight", true, false) ||
            lin(m, L.q_w, p + "self_attn.q_proj.weight", true, false) || lin(m, L.k_w, p + "self_attn.k_proj.weight", true, false) ||
            lin(m, L.v_w, p + "self_attn.v_proj.weight", true, false) || lin(m, L.o_w, p + "self_attn.o_proj.weight", true, false) ||
            lin(m, L.relk, p + "self_attn.relative_k_proj.weight", true, false) ||
            lin(m, L.pw1_w, p + "conv.pointwise_conv1.weight", true, false) || lin(m, L.pw2_w, p + "conv.pointwise_conv2.weight", true, false) ||
            finish_qkv(m, L))
            return -1;
    }
    m.ffn_dim = m.layers[0].ff1_w1.n;
    // tiles for the persistent few-row kernel: cache-aware streaming needs causal convs and the LayerNorm conv norm
    m.fr_stream = m.causal && !bn && m.d_model <= 1024 && m.d_model % 64 == 0 && fr_attn_fits(m.d_head);
    for (const EncLayer &L : m.layers)
        for (const QWeight *w : {&L.ff1_w1, &L.ff1_w2, &L.ff2_w1, &L.ff2_w2, &L.q_w, &L.k_w, &L.v_w, &L.o_w, &L.pw1_w, &L.pw2_w})
            m.fr_stream = m.fr_stream && fr_can_tile(*w) && w->n % 8 == 0;
    if (m.fr_stream)
        for (EncLayer &L : m.layers) {
            L.t_ff1a = m.fr_tiles({&L.ff1_w1}); L.t_ff1b = m.fr_tiles({&L.ff1_w2}); L.t_qkv = m.fr_tiles({&L.q_w, &L.k_w, &L.v_w});
            L.t_o = m.fr_tiles({&L.o_w}); L.t_pw1 = m.fr_tiles({&L.pw1_w}, true); L.t_pw2 = m.fr_tiles({&L.pw2_w});
            L.t_ff2a = m.fr_tiles({&L.ff2_w1}); L.t_ff2b = m.fr_tiles({&L.ff2_w2});
            if (!L.t_ff1a || !L.t_ff1b || !L.t_qkv || !L.t_o || !L.t_pw1 || !L.t_pw2 || !L.t_ff2a || !L.t_ff2b) return -1;
        }
    m.d_out = m.d_model;
    if (m.cfg.a8) {
        for (int li = 0; li < nl; li++) {
            const EncLayer &L = m.layers[li];
            const QWeight *ws[10] = {&L.ff1_w1, &L.ff1_w2, &L.ff2_w1, &L.ff2_w2, &L.q_w, &L.k_w, &L.v_w, &L.o_w, &L.pw1_w, &L.pw2_w};
            for (const QWeight *w : ws)
                if (!m.a8_ok(*w)) {
                    set_error("a8 mode: the linears of encoder layer %d must be reference-native int8 [n,k] with k %% 128 == 0 (got format %d, k=%d)", li, w->fmt, w->k);
                    return -1;
                }
        }
        m.a8_layers = true;
    }
    if (find(m, "encoder_projector.weight")) {
        if (lin(m, m.encproj, "encoder_projector.weight", true, false)) return -1;
        m.has_encproj = true;
        m.d_out = m.encproj.n;
    }
    if (const HostTensor *p1 = find(m, "prompt_projector.linear_1.weight")) {
        // Nemotron-style prompt MLP (mynah_asr_encoder_init, src/encoder.c:65-77,173-176): linear_1 is [inter, d + num_prompts]
        const HostTensor *b1 = find(m, "prompt_projector.linear_1.bias"), *p2 = find(m, "prompt_projector.linear_2.weight");
        const int d = m.d_model;
        if (!m.has_encproj || !b1 || !p2 || p1->fmt != FMT_F32 || b1->fmt != FMT_F32 || p1->shape.size() != 2 || (int)p1->shape[1] <= d) {
            set_error("prompt_projector needs f32 linear_1 [inter, d + prompts] with its bias, linear_2 and an encoder_projector"); return -1;
        }
        const int di = (int)p1->shape[0], dcat = (int)p1->shape[1], np = dcat - d;
        if (di % 64) { set_error("prompt_projector width %d must be a multiple of 64", di); return -1; }
        const float *w1 = (const float *)p1->data, *bb = (const float *)b1->data;
        std::vector<float> main((size_t)di * d), table((size_t)np * di);
        for (int i = 0; i < di; i++) {
            memcpy(&main[(size_t)i * d], w1 + (size_t)i * dcat, (size_t)d * sizeof(float));
            // the reference adds b1 to (x W^T + W[:, d + p]); the sum of the two constants first differs by an ulp at most
            for (int p = 0; p < np; p++) table[(size_t)p * di + i] = w1[(size_t)i * dcat + d + p] + bb[i];
        }
        if (m.upload_weight(m.prompt_l1, FMT_F32, main.data(), nullptr, di, d, true, false)) return -1;
        m.prompt_bias1 = m.upload_f32(table.data(), table.size());
        if (!m.prompt_bias1 || lin(m, m.prompt_l2, "prompt_projector.linear_2.weight", true, false)) return -1;
        if (!m.prompt_l2.bias || m.prompt_l2.n != d || m.prompt_l2.k != di) { set_error("prompt_projector.linear_2 must be [d, inter] with a bias"); return -1; }
        m.has_prompt = true; m.num_prompts = np; m.prompt_inter = di;
    }
    if (find(m, "ctc_head.weight")) {
        if (lin(m, m.ctc_head, "ctc_head.weight", true, false)) return -1;
        if (!m.ctc_head.bias) { set_error("missing ctc_head.bias"); return -1; }
        m.has_ctc = true;
        m.ctc_vocab = m.ctc_head.n;
    }
    if (const HostTensor *e = find(m, "decoder.embedding.weight")) {
        m.vocab = (int)e->shape[0]; m.pred_hidden = (int)e->shape[1];
        m.emb = f32dev(m, "decoder.embedding.weight", true, &err);
        if (m.emb) {                       // the same table as fp16 (hi, lo) planes: LSTM inputs are copied, not converted
            const size_t ne = (size_t)m.vocab * m.pred_hidden;
            m.emb_planes.hi = (__half *)m.dev_alloc(ne * 2); m.emb_planes.lo = (__half *)m.dev_alloc(ne * 2);
            if (!m.emb_planes.hi || !m.emb_planes.lo || split_to_h16(m.emb, m.emb_planes.hi, m.emb_planes.lo, ne, m.stream, m.status)) return -1;
        }
        m.proj_b = f32dev(m, "decoder.decoder_projector.bias", true, &err);
        m.head_b = f32dev(m, "joint.head.bias", true, &err);
        int n = 0;
        const int Hh = m.pred_hidden;
        for (; n < DEC_MAX_LAYERS; n++) {
            const std::string s = std::to_string(n);
            const HostTensor *wi = find(m, "decoder.lstm.weight_ih_l" + s), *wh = find(m, "decoder.lstm.weight_hh_l" + s);
            if (!wi) break;
            if (!wh || wi->fmt != FMT_F32 || wh->fmt != FMT_F32 || (int)wi->nelem() != 4 * Hh * Hh || (int)wh->nelem() != 4 * Hh * Hh) {
                set_error("LSTM layer %d is incomplete or has an unexpected shape", n); return -1;
            }
            m.b_ih[n] = f32dev(m, "decoder.lstm.bias_ih_l" + s, true, &err);
            m.b_hh[n] = f32dev(m, "decoder.lstm.bias_hh_l" + s, true, &err);
            // [W_ih | W_hh] side by side so one contraction over [input ; h] gives the gate pre-activations
            std::vector<float> cat((size_t)4 * Hh * 2 * Hh);
            for (int r = 0; r < 4 * Hh; r++) {
                memcpy(&cat[(size_t)r * 2 * Hh], (const float *)wi->data + (size_t)r * Hh, Hh * sizeof(float));
                memcpy(&cat[(size_t)r * 2 * Hh + Hh], (const float *)wh->data + (size_t)r * Hh, Hh * sizeof(float));
            }
            if (m.upload_weight(m.wcat[n], FMT_F32, cat.data(), nullptr, 4 * Hh, 2 * Hh, true, false)) return -1;
        }
        if (err) return -1;
        if (n == 0 || m.pred_hidden > 1024 || m.pred_hidden % 32) { set_error("unsupported prediction network (layers %d, hidden %d)", n, m.pred_hidden); return -1; }
        m.pred_layers = n;
        if (lin(m, m.dec_proj, "decoder.decoder_projector.weight", true, false)) return -1;
        if (lin(m, m.head, "joint.head.weight", true, false)) return -1;
        if (m.head.n != m.vocab + m.cfg.n_durations) { set_error("joint head has %d rows, expected vocab %d + %d durations", m.head.n, m.vocab, m.cfg.n_durations); return -1; }
        if (m.d_out != m.pred_hidden) { set_error("encoder output width %d != prediction hidden %d", m.d_out, m.pred_hidden); return -1; }
        m.has_dec = true;
    }
    if (const HostTensor *e = find(m, "aed.embedding.weight")) {
        // mynah_asr_aed_init (src/decoder_aed.c:50-113)
        if (e->fmt != FMT_F32 || e->shape.size() != 2) { set_error("aed.embedding.weight must be f32 [vocab, d]"); return -1; }
        m.aed_vocab = (int)e->shape[0]; m.aed_d = (int)e->shape[1];
        m.aed_heads = m.cfg.aed_heads > 0 ? m.cfg.aed_heads : 8;
        if (m.aed_d % m.aed_heads || m.aed_d % 64) { set_error("AED width %d must be a multiple of 64 and of its %d heads", m.aed_d, m.aed_heads); return -1; }
        const HostTensor *pe = find(m, "aed.pos_enc");
        if (!pe || pe->shape.size() != 2 || (int)pe->shape[1] != m.aed_d) { set_error("missing or misshapen aed.pos_enc"); return -1; }
        m.aed_max_seq = (int)pe->shape[0];
        m.aed_emb = f32dev(m, "aed.embedding.weight", true, &err);
        m.aed_pos = f32dev(m, "aed.pos_enc", true, &err);
        m.aed_embln_w = f32dev(m, "aed.emb_norm.weight", true, &err); m.aed_embln_b = f32dev(m, "aed.emb_norm.bias", true, &err);
        m.aed_fin_w = f32dev(m, "aed.final_norm.weight", true, &err); m.aed_fin_b = f32dev(m, "aed.final_norm.bias", true, &err);
        if (err) return -1;
        if (lin(m, m.aed_head, "aed.head.weight", true, false)) return -1;
        m.aed_head_b = m.aed_head.bias;
        if (!m.aed_head_b) { set_error("missing aed.head.bias"); return -1; }
        if (find(m, "enc_dec_proj.weight")) {
            if (lin(m, m.aed_proj, "enc_dec_proj.weight", true, false)) return -1;
            m.aed_proj_b = m.aed_proj.bias;
            m.has_aed_proj = true;
            if (m.aed_proj.n != m.aed_d || m.aed_proj.k != m.d_out) { set_error("enc_dec_proj is [%d,%d], expected [%d,%d]", m.aed_proj.n, m.aed_proj.k, m.aed_d, m.d_out); return -1; }
        } else if (m.d_out != m.aed_d) { set_error("encoder output width %d != AED width %d and no enc_dec_proj", m.d_out, m.aed_d); return -1; }
        int nl = 0;
        while (find(m, "aed.layers." + std::to_string(nl) + ".ln_self.weight")) nl++;
        if (nl == 0) { set_error("AED decoder without layers"); return -1; }
        m.aed_layers.resize(nl);
        for (int li = 0; li < nl; li++) {
            AedLayer &A = m.aed_layers[li];
            const std::string p = "aed.layers." + std::to_string(li) + ".";
            A.ln_self_w = f32dev(m, p + "ln_self.weight", true, &err); A.ln_self_b = f32dev(m, p + "ln_self.bias", true, &err);
            A.ln_cross_w = f32dev(m, p + "ln_cross.weight", true, &err); A.ln_cross_b = f32dev(m, p + "ln_cross.bias", true, &err);
            A.ln_ffn_w = f32dev(m, p + "ln_ffn.weight", true, &err); A.ln_ffn_b = f32dev(m, p + "ln_ffn.bias", true, &err);
            if (err) return -1;
            if (lin_cat(m, A.sqkv, &A.sqkv_b, {p + "self_attn.q_proj", p + "self_attn.k_proj", p + "self_attn.v_proj"}) ||
                lin_cat(m, A.ckv, &A.ckv_b, {p + "cross_attn.k_proj", p + "cross_attn.v_proj"}) ||
                lin_cat(m, A.so, &A.so_b, {p + "self_attn.o_proj"}) || lin_cat(m, A.cq, &A.cq_b, {p + "cross_attn.q_proj"}) ||
                lin_cat(m, A.co, &A.co_b, {p + "cross_attn.o_proj"}) || lin_cat(m, A.ff1, &A.ff1_b, {p + "ffn.linear1"}) ||
                lin_cat(m, A.ff2, &A.ff2_b, {p + "ffn.linear2"}))
                return -1;
            if (A.sqkv.n != 3 * m.aed_d || A.ckv.n != 2 * m.aed_d || A.sqkv.k != m.aed_d || A.ff2.n != m.aed_d || A.ff1.n % 64) {
                set_error("AED layer %d has unexpected shapes", li); return -1;
            }
        }
        m.aed_ffn = m.aed_layers[0].ff1.n;
        m.fr_aed = m.aed_d <= 1024 && fr_attn_fits(m.aed_d / m.aed_heads) && fr_can_tile(m.aed_head);
        for (const AedLayer &A : m.aed_layers)
            for (const QWeight *w : {&A.sqkv, &A.so, &A.cq, &A.co, &A.ff1, &A.ff2}) m.fr_aed = m.fr_aed && fr_can_tile(*w);
        if (m.fr_aed) {
            for (AedLayer &A : m.aed_layers) {
                A.t_sqkv = m.fr_tiles({&A.sqkv}); A.t_so = m.fr_tiles({&A.so}); A.t_cq = m.fr_tiles({&A.cq});
                A.t_co = m.fr_tiles({&A.co}); A.t_ff1 = m.fr_tiles({&A.ff1}); A.t_ff2 = m.fr_tiles({&A.ff2});
                if (!A.t_sqkv || !A.t_so || !A.t_cq || !A.t_co || !A.t_ff1 || !A.t_ff2) return -1;
            }
            m.t_aed_head = m.fr_tiles({&m.aed_head});
            if (!m.t_aed_head) return -1;
        }
        m.has_aed = true;
    }
    m.host.clear();
    MB_CUDA(cudaDeviceSynchronize());
    if (m.check_status("model_finalize (a weight does not fit the fp16 operand planes)")) return -1;
    m.release_load_buffers();
    m.load_seconds += std::chrono::duration<double>(std::chrono::steady_clock::now() - t_load0).count();
    m.finalized = true;
    return 0;
}

void mynah_b200_model_free(mynah_b200_model *h) { delete h; }

int mynah_b200_model_set_max_contexts(mynah_b200_model *h, int n) {
    if (!h || n < 1 || n > 64) { set_error("model_set_max_contexts: 1..64"); return -1; }
    std::lock_guard<std::mutex> lk(h->pool_mu);
    if (n < h->n_ctx()) { set_error("model_set_max_contexts: %d contexts already exist", h->n_ctx()); return -1; }
    h->max_ctx = n;
    return 0;
}

int mynah_b200_model_set_strict(mynah_b200_model *h, int strict) {
    if (!h) { set_error("model_set_strict: null model"); return -1; }
    with_all_contexts_idle(h, [&](Model &c) { c.cfg.strict = strict ? 1 : 0; });
    return 0;
}

void mynah_b200_model_dims(const mynah_b200_model *h, int *dims) {
    const Model &m = h->m;
    dims[0] = m.d_model; dims[1] = m.n_layers; dims[2] = m.n_heads; dims[3] = m.ffn_dim;
    dims[4] = m.conv_k; dims[5] = m.d_out; dims[6] = m.causal; dims[7] = m.channels;
}

void *mynah_b200_model_stream(mynah_b200_model *h) { return h ? (void *)h->m.stream : nullptr; }

void mynah_b200_model_load_stats(const mynah_b200_model *h, double *seconds, double *host_bytes, double *device_bytes) {
    if (!h) return;
    double dev = 0.0;
    for (const auto &sl : h->m.slabs) dev += (double)sl.off;
    if (seconds) *seconds = h->m.load_seconds;
    if (host_bytes) *host_bytes = (double)h->m.load_bytes;
    if (device_bytes) *device_bytes = dev;
}

}  // extern "C"

// -------------------------------------------------------------- workspace sizes
static size_t enc_bytes(const Model &m, size_t M, size_t max_len) {
    const size_t rk_rows = 2 * max_len + 1;
    return M * ((size_t)m.d_model * 44 + (size_t)m.ffn_dim * 4) +
           rk_rows * m.d_model * (4 + 2 * (size_t)m.rk_layers((int)rk_rows, m.n_layers)) + (1 << 20) +
           (m.a8_layers ? M * ((size_t)m.d_model + 5 * (size_t)m.ffn_dim + 64) + 4096 : 0);
}
static size_t stage_bytes(int batch) { return (size_t)batch * (sizeof(FrontItem) + 16) + 4096; }
static size_t dec_bytes(const Model &m, int max_len) {
    const size_t B = DEC_MAX_B;
    return (size_t)max_len * m.cfg.max_symbols * B * 8 + B * 148 * 8 * 16 + 4 * (size_t)DEC_MAX_LAYERS * B * 1024 * 4 + B * (size_t)m.pred_hidden * 4 + (1 << 20);
}

extern "C" {

float *mynah_b200_log_mel(mynah_b200_model *h, const float *audio, size_t n, int *n_frames, int *valid_frames) {
    if (!h || !h->m.finalized || (!audio && n)) { set_error("log_mel: bad argument"); return nullptr; }
    Lease lease(h);
    Model &m = lease.model();
    const int hop = m.cfg.hop_length, T = 1 + (int)(n / hop), valid = (int)(n / hop), nm = m.cfg.n_mels;
    if (m.ws.reserve(n * 4 + (size_t)T * nm * 4 + (1 << 20))) return nullptr;
    m.ws.reset();
    float *a = m.ws.get<float>(n ? n : 1), *f = m.ws.get<float>((size_t)T * nm);
    if (!a || !f) return nullptr;
    MB_CUDA_NULL(cudaMemcpyAsync(a, audio, n * 4, cudaMemcpyHostToDevice, m.stream));
    if (m.log_mel(a, n, f, T, valid)) return nullptr;
    float *out = (float *)malloc((size_t)T * nm * sizeof(float));
    if (!out) { set_error("out of host memory"); return nullptr; }
    MB_CUDA_NULL(cudaMemcpyAsync(out, f, (size_t)T * nm * 4, cudaMemcpyDeviceToHost, m.stream));
    MB_CUDA_NULL(cudaStreamSynchronize(m.stream));
    *n_frames = T; *valid_frames = valid;
    return out;
}

float *mynah_b200_subsampling_forward(mynah_b200_model *h, const float *feats, int T, int n_mels, int *t_out) {
    if (!h || !h->m.finalized || !feats || T <= 0 || n_mels != h->m.cfg.n_mels) { set_error("subsampling_forward: bad argument"); return nullptr; }
    Lease lease(h);
    Model &m = lease.model();
    const int T3 = m.enc_len(T);
    if (m.ws.reserve(m.front_bytes(nullptr, &T, 1, false, true) + (size_t)T3 * m.d_model * 4 + (1 << 20)) || m.host_stage.begin(stage_bytes(1))) return nullptr;
    m.ws.reset();
    float *x = m.ws.get<float>((size_t)T3 * m.d_model);
    std::vector<int> lens;
    if (!x || m.front_end(nullptr, nullptr, &feats, &T, 1, true, x, lens) || m.check_status("subsampling")) return nullptr;
    const int t = lens[0];
    float *out = (float *)malloc((size_t)t * m.d_model * sizeof(float));
    if (!out) { set_error("out of host memory"); return nullptr; }
    MB_CUDA_NULL(cudaMemcpyAsync(out, x, (size_t)t * m.d_model * 4, cudaMemcpyDeviceToHost, m.stream));
    MB_CUDA_NULL(cudaStreamSynchronize(m.stream));
    *t_out = t;
    return out;
}

int mynah_b200_encoder_layer(mynah_b200_model *h, int li, float *x, int T, int left, int right) {
    if (!h || !h->m.finalized || !x || T <= 0 || li < 0 || li >= h->m.n_layers) { set_error("encoder_layer: bad argument"); return -1; }
    Lease lease(h);
    Model &m = lease.model();
    if (m.ws.reserve(enc_bytes(m, T, T) + (size_t)T * m.d_model * 4) || m.host_stage.begin(stage_bytes(1))) return -1;
    m.ws.reset();
    float *xd = m.ws.get<float>((size_t)T * m.d_model);
    MB_CUDA(cudaMemcpyAsync(xd, x, (size_t)T * m.d_model * 4, cudaMemcpyHostToDevice, m.stream));
    std::vector<int> lens{T};
    if (m.encoder_layers(xd, lens, left, right, li, 1) || m.check_status("encoder_layer")) return -1;
    MB_CUDA(cudaMemcpyAsync(x, xd, (size_t)T * m.d_model * 4, cudaMemcpyDeviceToHost, m.stream));
    MB_CUDA(cudaStreamSynchronize(m.stream));
    return 0;
}

int mynah_b200_encoder_forward_batch(mynah_b200_model *h, const float *const *feats, const int *t_mel, int batch,
                                     int n_mels, const int *prompt_ids, int left, int right, float **outs, int *t_outs) {
    if (!h || !h->m.finalized || batch <= 0 || n_mels != h->m.cfg.n_mels) { set_error("encoder_forward_batch: bad argument"); return -1; }
    Lease lease(h);
    Model &m = lease.model();
    size_t M = 0, max_len = 0;
    for (int b = 0; b < batch; b++) {
        const size_t t = t_mel[b] > 0 ? m.enc_len(t_mel[b]) : 0;
        M += t;
        if (t > max_len) max_len = t;
    }
    if (m.ws.reserve(m.front_bytes(nullptr, t_mel, batch, false, true) + enc_bytes(m, M, max_len) + M * ((size_t)m.d_model + m.d_out) * 4 + (1 << 20)) ||
        m.host_stage.begin(stage_bytes(batch)))
        return -1;
    m.ws.reset();
    std::vector<int> lens;
    float *x = m.ws.get<float>((M ? M : 1) * m.d_model), *y = m.ws.get<float>((M ? M : 1) * m.d_out);
    if (!x || !y) return -1;
    if (m.front_end(nullptr, nullptr, feats, t_mel, batch, true, x, lens) || m.encoder_layers(x, lens, left, right, 0, m.n_layers)) return -1;
    if (m.encoder_post(x, lens, prompt_ids, y) || m.check_status("encoder_forward_batch")) return -1;
    size_t off = 0;
    std::vector<CopyOut> parts;
    for (int b = 0; b < batch; b++) {
        t_outs[b] = lens[b];
        outs[b] = (float *)malloc((size_t)(lens[b] ? lens[b] : 1) * m.d_out * sizeof(float));
        if (!outs[b]) { set_error("out of host memory"); return -1; }
        parts.push_back(CopyOut{outs[b], y + off * m.d_out, (size_t)lens[b] * m.d_out * 4});
        off += lens[b];
    }
    if (copy_out(parts, m.stream)) return -1;
    MB_CUDA(cudaStreamSynchronize(m.stream));
    lease.idle();
    return 0;
}

static float *forward_one(mynah_b200_model *h, const float *feats, int t_mel, int n_mels, int prompt_id, int left, int right,
                          int raw, int *t_out) {
    if (!h || !h->m.finalized || !feats || t_mel <= 0 || n_mels != h->m.cfg.n_mels) { set_error("encoder_forward: bad argument"); return nullptr; }
    Lease lease(h);
    Model &m = lease.model();
    const size_t M = m.enc_len(t_mel);
    if (m.ws.reserve(m.front_bytes(nullptr, &t_mel, 1, false, true) + enc_bytes(m, M, M) + M * ((size_t)m.d_model + m.d_out) * 4 + (1 << 20)) ||
        m.host_stage.begin(stage_bytes(1)))
        return nullptr;
    m.ws.reset();
    float *x = m.ws.get<float>(M * m.d_model), *y = m.ws.get<float>(M * m.d_out);
    if (!x || !y) return nullptr;
    std::vector<int> lens;
    if (m.front_end(nullptr, nullptr, &feats, &t_mel, 1, true, x, lens) || m.encoder_layers(x, lens, left, right, 0, m.n_layers)) return nullptr;
    const int wout = raw ? m.d_model : m.d_out;
    if (!raw && m.encoder_post(x, lens, &prompt_id, y)) return nullptr;
    if (m.check_status("encoder_forward")) return nullptr;
    float *out = (float *)malloc(M * wout * sizeof(float));
    if (!out) { set_error("out of host memory"); return nullptr; }
    if (copy_out(out, raw ? x : y, M * wout * 4, m.stream)) return nullptr;
    MB_CUDA_NULL(cudaStreamSynchronize(m.stream));
    lease.idle();
    *t_out = (int)M;
    return out;
}

float *mynah_b200_encoder_forward(mynah_b200_model *h, const float *feats, int t_mel, int n_mels, int prompt_id,
                                  int left, int right, int *t_out) {
    return forward_one(h, feats, t_mel, n_mels, prompt_id, left, right, 0, t_out);
}
float *mynah_b200_encoder_forward_raw(mynah_b200_model *h, const float *feats, int t_mel, int n_mels, int left,
                                      int right, int *t_out) {
    return forward_one(h, feats, t_mel, n_mels, 0, left, right, 1, t_out);
}

int mynah_b200_ctc_decode(mynah_b200_model *h, const float *enc_out, int T, int *tokens, int *frames, int cap) {
    if (!h || !h->m.finalized || !enc_out || T < 0) { set_error("ctc_decode: bad argument"); return -1; }
    Lease lease(h);
    Model &m = lease.model();
    if (T == 0) return 0;
    if (m.ws.reserve((size_t)T * (m.d_model * 8 + m.ctc_vocab * 4 + 8) + (1 << 20))) return -1;
    m.ws.reset();
    float *e = m.ws.get<float>((size_t)T * m.d_model);
    MB_CUDA(cudaMemcpyAsync(e, enc_out, (size_t)T * m.d_model * 4, cudaMemcpyHostToDevice, m.stream));
    std::vector<int> tk, fr;
    if (m.decode_ctc(e, T, tk, fr) || m.check_status("ctc_decode")) return -1;
    int n = 0;
    for (size_t i = 0; i < tk.size() && n < cap; i++, n++) { tokens[n] = tk[i]; if (frames) frames[n] = fr[i]; }
    return n;
}

int mynah_b200_greedy_decode(mynah_b200_model *h, const float *enc, int T, int *tokens, int *frames, int cap) {
    if (!h || !h->m.finalized || !enc || T < 0) { set_error("greedy_decode: bad argument"); return -1; }
    Lease lease(h);
    Model &m = lease.model();
    if (T == 0) return 0;
    if (m.ws.reserve((size_t)T * m.d_out * 4 + dec_bytes(m, T))) return -1;
    m.ws.reset();
    float *e = m.ws.get<float>((size_t)T * m.d_out);
    MB_CUDA(cudaMemcpyAsync(e, enc, (size_t)T * m.d_out * 4, cudaMemcpyHostToDevice, m.stream));
    std::vector<int> lens{T};
    std::vector<std::vector<int>> tk, fr;
    if (m.decode_greedy(e, lens, tk, fr) || m.check_status("greedy_decode")) return -1;
    int n = 0;
    for (size_t i = 0; i < tk[0].size() && n < cap; i++, n++) { tokens[n] = tk[0][i]; if (frames) frames[n] = fr[0][i]; }
    return n;
}

int mynah_b200_aed_decode_batch(mynah_b200_model *h, const float *const *encs, const int *Ts, int batch, const int *const *prompts,
                                const int *n_prompts, int eos, const int *caps, int **tokens, int *n_tokens) {
    if (!h || !h->m.finalized || !encs || !Ts || batch <= 0 || !prompts || !n_prompts || !caps || !tokens || !n_tokens) {
        set_error("aed_decode_batch: bad argument"); return -1;
    }
    Lease lease(h);
    Model &m = lease.model();
    if (!m.has_aed) { set_error("model has no AED decoder"); return -1; }
    size_t total = 0;
    int max_len = 0;
    std::vector<int> lens(Ts, Ts + batch), cp(caps, caps + batch);
    std::vector<std::vector<int>> pr(batch);
    for (int b = 0; b < batch; b++) {
        if (Ts[b] <= 0 || n_prompts[b] <= 0 || !prompts[b] || !encs[b]) { set_error("aed_decode_batch: utterance %d is empty or has no start token", b); return -1; }
        total += (size_t)Ts[b];
        pr[b].assign(prompts[b], prompts[b] + n_prompts[b]);
        const int ml = n_prompts[b] + (caps[b] > 0 ? caps[b] : 0);
        max_len = ml > max_len ? ml : max_len;
    }
    if (max_len > m.aed_max_seq) max_len = m.aed_max_seq;
    if (m.ws.reserve(total * m.d_out * 4 + m.aed_bytes((int)total, batch, max_len))) return -1;
    m.ws.reset();
    float *e = m.ws.get<float>(total * m.d_out);
    if (!e) return -1;
    size_t off = 0;
    for (int b = 0; b < batch; b++) {
        MB_CUDA(cudaMemcpyAsync(e + off * m.d_out, encs[b], (size_t)Ts[b] * m.d_out * 4, cudaMemcpyHostToDevice, m.stream));
        off += (size_t)Ts[b];
    }
    std::vector<std::vector<int>> tk;
    if (m.decode_aed(e, lens, pr, eos, cp, tk)) return -1;
    for (int b = 0; b < batch; b++) {
        n_tokens[b] = (int)tk[b].size();
        tokens[b] = (int *)malloc((tk[b].size() ? tk[b].size() : 1) * sizeof(int));
        if (!tokens[b]) { set_error("out of host memory"); return -1; }
        memcpy(tokens[b], tk[b].data(), tk[b].size() * sizeof(int));
    }
    return 0;
}

int mynah_b200_aed_decode(mynah_b200_model *h, const float *enc, int T, const int *prompt, int n_prompt, int eos, int *tokens, int cap) {
    if (!tokens || n_prompt <= 0 || !prompt) { set_error("aed_decode: bad argument (at least one start token is needed)"); return -1; }
    int *out = nullptr, n = 0;
    if (mynah_b200_aed_decode_batch(h, &enc, &T, 1, &prompt, &n_prompt, eos, &cap, &out, &n)) return -1;
    memcpy(tokens, out, (size_t)n * sizeof(int));
    free(out);
    return n;
}

void mynah_b200_batch_set_prompts(mynah_b200_batch *bt, const int *prompt_ids) {
    if (!bt) return;
    if (prompt_ids) bt->prompt_ids.assign(prompt_ids, prompt_ids + bt->batch); else bt->prompt_ids.clear();
}

void mynah_b200_batch_set_aed(mynah_b200_batch *bt, const int *prompt, int n_prompt, int eos, int max_gen_delta) {
    if (!bt) return;
    bt->aed_prompt.assign(prompt, prompt + (n_prompt > 0 ? n_prompt : 0));
    bt->aed_eos = eos; bt->aed_delta = max_gen_delta;
}

// ------------------------------------------------------------ CTC forced alignment
int mynah_b200_align_min_frames(const int *tokens, int n_tokens) { return tokens ? align_min_frames(tokens, n_tokens) : 0; }

int mynah_b200_align_ctc(const float *scores, int T, int V, const int *tokens, int n_tokens, int blank, int *t0, int *t1) {
    if (!scores || T <= 0 || V <= 0) { set_error("align_ctc: bad argument"); return -1; }
    if (!mynah_b200_available()) { set_error("align_ctc: no sm_100 device"); return -1; }
    float *d = nullptr;
    MB_CUDA(cudaMalloc((void **)&d, (size_t)T * V * sizeof(float)));
    int rc = -1;
    if (cudaMemcpy(d, scores, (size_t)T * V * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess)
        rc = align_ctc_device(d, T, V, tokens, n_tokens, blank, t0, t1, nullptr);
    else set_error("align_ctc: H2D copy failed");
    cudaFree(d);
    return rc;
}

int mynah_b200_ctc_align(mynah_b200_model *h, const float *enc_out, int T, const int *tokens, int n_tokens, int *t0, int *t1) {
    if (!h || !h->m.finalized || !enc_out || T <= 0 || !tokens || n_tokens <= 0) { set_error("ctc_align: bad argument"); return -1; }
    Lease lease(h);
    Model &m = lease.model();
    if (!m.has_ctc) { set_error("ctc_align: model has no CTC head"); return -1; }
    const int V = m.ctc_vocab, d = m.d_model;
    if (m.ws.reserve((size_t)T * ((size_t)d * 8 + (size_t)V * 4 + 8) + (1 << 20))) return -1;
    m.ws.reset();
    float *e = m.ws.get<float>((size_t)T * d), *logits = m.ws.get<float>((size_t)T * V);
    H16 hp = m.ws.planes((size_t)T * d);
    if (!e || !logits || !hp.lo) return -1;
    MB_CUDA(cudaMemcpyAsync(e, enc_out, (size_t)T * d * 4, cudaMemcpyHostToDevice, m.stream));
    if (split_to_h16(e, hp.hi, hp.lo, (size_t)T * d, m.stream, m.status)) return -1;
    note_launch();
    GemmEpilogue ep;
    memset(&ep, 0, sizeof(ep));
    ep.mode = OUT_F32; ep.act = ACT_NONE; ep.alpha = 1.f; ep.bias = m.ctc_head.bias; ep.out = logits; ep.ldo = V;
    if (m.gemm(hp, d, m.ctc_head, ep, T)) return -1;
    if (m.check_status("ctc_align")) return -1;
    return align_ctc_device(logits, T, V, tokens, n_tokens, V - 1, t0, t1, m.stream);
}

// ------------------------------------------------------------ cache-aware streaming
mynah_b200_stream_group *mynah_b200_stream_open(mynah_b200_model *h, int n_streams, int left_ctx, int right_ctx) {
    if (!h || !h->m.finalized) { set_error("stream_open: bad argument"); return nullptr; }
    Lease lease(h);
    Model &m = lease.model();
    mynah_b200_stream_group *g = new mynah_b200_stream_group();
    g->model = h;
    g->ctx = lease.index();
    if (m.stream_open(g->st, n_streams, left_ctx, right_ctx)) { m.stream_close(g->st); delete g; return nullptr; }
    return g;
}

void mynah_b200_stream_close(mynah_b200_stream_group *g) {
    if (!g) return;
    { Lease lease(g->model, g->ctx); lease.model().stream_close(g->st); }
    delete g;
}

int mynah_b200_stream_set_prompts(mynah_b200_stream_group *g, const int *prompt_ids) {
    if (!g || !prompt_ids) { set_error("stream_set_prompts: bad argument"); return -1; }
    Lease lease(g->model, g->ctx);
    Model &m = lease.model();
    if (g->st.exec) { set_error("stream_set_prompts: set the prompts before the first step"); return -1; }
    g->st.prompt_ids.assign(prompt_ids, prompt_ids + g->st.S);
    return 0;
}

int mynah_b200_stream_need(const mynah_b200_stream_group *g) { return g ? g->model->m.stream_need(g->st) : -1; }

int mynah_b200_stream_step_device(mynah_b200_stream_group *g, const float *mel_dev, int n_mel, int is_last, float *out_dev) {
    if (!g || !mel_dev || !out_dev) { set_error("stream_step: bad argument"); return -1; }
    Lease lease(g->model, g->ctx);
    Model &m = lease.model();
    if (n_mel != m.stream_need(g->st) && !is_last) { set_error("stream_step: %d mel frames given, %d needed", n_mel, m.stream_need(g->st)); return -1; }
    if (m.ws.reserve(m.stream_bytes(g->st, n_mel))) return -1;
    m.ws.reset();
    const int q = m.stream_step(g->st, mel_dev, n_mel, is_last, out_dev);
    if (q < 0 || m.check_status("stream_step")) return -1;
    lease.idle();
    return q;
}

int mynah_b200_stream_step(mynah_b200_stream_group *g, const float *mel, int n_mel, int is_last, float *out) {
    if (!g || !mel || !out || n_mel <= 0) { set_error("stream_step: bad argument"); return -1; }
    Lease lease(g->model, g->ctx);
    Model &m = lease.model();
    if (n_mel != m.stream_need(g->st) && !is_last) { set_error("stream_step: %d mel frames given, %d needed", n_mel, m.stream_need(g->st)); return -1; }
    const size_t S = g->st.S, nin = S * n_mel * m.cfg.n_mels, nout = S * (g->st.q + 2) * m.d_out;
    if (m.ws.reserve(m.stream_bytes(g->st, n_mel) + (nin + nout) * 4 + 4096)) return -1;
    m.ws.reset();
    float *md = m.ws.get<float>(nin), *od = m.ws.get<float>(nout);
    if (!md || !od) return -1;
    if (copy_in(md, mel, nin * 4, m.stream)) return -1;
    const int q = m.stream_step(g->st, md, n_mel, is_last, od);
    if (q < 0) return -1;
    if (copy_out(out, od, S * q * m.d_out * 4, m.stream)) return -1;
    MB_CUDA(cudaStreamSynchronize(m.stream));
    if (m.check_status("stream_step")) return -1;
    lease.idle();
    return q;
}

int mynah_b200_stream_mel_feed(mynah_b200_stream_group *g, const float *audio, int n, int finish, float *out, int cap_frames) {
    if (!g || !out) { set_error("stream_mel_feed: bad argument"); return -1; }
    Lease lease(g->model, g->ctx);
    Model &m = lease.model();
    if (m.ws.reserve((size_t)g->st.S * (size_t)(cap_frames > 0 ? cap_frames : 1) * m.cfg.n_mels * 4 + (1 << 20))) return -1;
    m.ws.reset();
    return m.stream_mel_feed(g->st, audio, n, finish, out, cap_frames);
}

int mynah_b200_stream_step_decode(mynah_b200_stream_group *g, const float *mel, int n_mel, int is_last, int **tokens,
                                  int **frames, int *n_tokens) {
    if (!g || !mel || n_mel <= 0 || !tokens || !n_tokens) { set_error("stream_step_decode: bad argument"); return -1; }
    Lease lease(g->model, g->ctx);
    Model &m = lease.model();
    if (!m.has_dec) { set_error("stream_step_decode: model has no transducer decoder"); return -1; }
    if (n_mel != m.stream_need(g->st) && !is_last) { set_error("stream_step: %d mel frames given, %d needed", n_mel, m.stream_need(g->st)); return -1; }
    const size_t S = g->st.S, nin = S * n_mel * m.cfg.n_mels, nout = S * (g->st.q + 2) * m.d_out;
    const size_t nw = (size_t)(m.vocab + m.cfg.n_durations + 15) / 16, cap = (size_t)(g->st.q + 2) * m.cfg.max_symbols;
    const size_t decb = S * (24 + 4 * nw + 2 * cap) * 4 + ((S + 15) / 16) * (1024 + (size_t)DEC_MAX_B * m.pred_hidden * 4) + (1 << 20);
    if (m.ws.reserve(m.stream_bytes(g->st, n_mel) + (nin + nout) * 4 + decb + 4096)) return -1;
    m.ws.reset();
    float *md = m.ws.get<float>(nin), *od = m.ws.get<float>(nout);
    if (!md || !od) return -1;
    if (copy_in(md, mel, nin * 4, m.stream)) return -1;
    const int q = m.stream_step(g->st, md, n_mel, is_last, od);
    if (q < 0) return -1;
    std::vector<std::vector<int>> tk, fr;
    if (m.stream_decode(g->st, od, q, tk, fr) || m.check_status("stream_step_decode")) return -1;
    lease.idle();
    for (size_t s = 0; s < S; s++) {
        n_tokens[s] = (int)tk[s].size();
        tokens[s] = (int *)malloc((tk[s].size() ? tk[s].size() : 1) * sizeof(int));
        if (frames) frames[s] = (int *)malloc((tk[s].size() ? tk[s].size() : 1) * sizeof(int));
        if (!tokens[s] || (frames && !frames[s])) { set_error("out of host memory"); return -1; }
        memcpy(tokens[s], tk[s].data(), tk[s].size() * sizeof(int));
        if (frames) memcpy(frames[s], fr[s].data(), fr[s].size() * sizeof(int));
    }
    return q;
}

// ------------------------------------------------------------ resident pipeline
mynah_b200_batch *mynah_b200_batch_upload(mynah_b200_model *h, const float *const *audio, const size_t *n_samples, int batch) {
    if (!h || !h->m.finalized || batch <= 0) { set_error("batch_upload: bad argument"); return nullptr; }
    mynah_b200_batch *bt = new mynah_b200_batch();
    bt->batch = batch;
    bt->audio.assign(batch, nullptr);
    bt->n_samples.assign(n_samples, n_samples + batch);
    for (int b = 0; b < batch; b++) {
        if (cudaMalloc(&bt->audio[b], (n_samples[b] ? n_samples[b] : 1) * sizeof(float)) != cudaSuccess) {
            set_error("batch_upload: cudaMalloc failed"); mynah_b200_batch_free(bt); return nullptr;
        }
        cudaMemcpyAsync(bt->audio[b], audio[b], n_samples[b] * sizeof(float), cudaMemcpyHostToDevice, h->m.stream);
    }
    cudaStreamSynchronize(h->m.stream);
    return bt;
}

void mynah_b200_batch_free(mynah_b200_batch *bt) {
    if (!bt) return;
    for (float *p : bt->audio) if (p) cudaFree(p);
    delete bt;
}

// Whole path for one batch. audio_dev: utterances already on the device, or null with
// audio_host set: then the audio is copied into the workspace arena first (no allocation
// on the hot path). Caller holds the model lock.
static int run_batch_locked(Model &m, mynah_b200_batch *bt, const float *const *audio_dev, const float *const *audio_host,
                            int decoder) {
    const int B = bt->batch, hop = m.cfg.hop_length;
    size_t M = 0;
    int max_len = 0;
    std::vector<int> valid(B);
    for (int b = 0; b < B; b++) {
        valid[b] = (int)(bt->n_samples[b] / hop);
        const int t = valid[b] > 0 ? m.enc_len(valid[b]) : 0;
        M += t; if (t > max_len) max_len = t;
    }
    if (decoder == 2 && (!m.has_aed || bt->aed_prompt.empty())) { set_error("batch_run: AED decoding needs an AED model and mynah_b200_batch_set_aed"); return -1; }
    int aed_len = (int)bt->aed_prompt.size() + max_len + bt->aed_delta;
    if (decoder == 2 && aed_len > m.aed_max_seq) aed_len = m.aed_max_seq;
    const size_t decb = decoder == 1 ? M * ((size_t)m.d_model * 4 + (size_t)m.ctc_vocab * 4 + 8)
                      : decoder == 2 ? m.aed_bytes((int)M, B, aed_len) : dec_bytes(m, max_len);
    if (m.ws.reserve(m.front_bytes(bt->n_samples.data(), valid.data(), B, true, audio_host != nullptr) + enc_bytes(m, M, max_len) +
                     M * ((size_t)m.d_model + m.d_out) * 4 + decb + (4 << 20)) ||
        m.host_stage.begin(stage_bytes(B)))
        return -1;
    m.ws.reset();
    float *x = m.ws.get<float>((M ? M : 1) * m.d_model), *y = m.ws.get<float>((M ? M : 1) * m.d_out);
    if (!x || !y) return -1;
    std::vector<int> lens;
    if (m.front_end(audio_host ? audio_host : audio_dev, bt->n_samples.data(), nullptr, valid.data(), B, audio_host != nullptr, x, lens) ||
        m.encoder_layers(x, lens, m.cfg.left_ctx, m.cfg.right_ctx, 0, m.n_layers))
        return -1;
    bt->tokens.assign(B, {}); bt->frames.assign(B, {});
    if (decoder == 1) {
        size_t off = 0;
        for (int b = 0; b < B; b++) {      // CTC works on the raw encoder output (engine raw_encoder = 1)
            if (m.decode_ctc(x + off * m.d_model, lens[b], bt->tokens[b], bt->frames[b])) return -1;
            off += lens[b];
        }
    } else if (decoder == 2) {
        // AED engine: projected encoder output, generation budget T + max_gen_delta per utterance
        // (eng_decode_aed, src/mynah_asr.c:147-160, without timestamp tokens)
        if (m.encoder_post(x, lens, bt->prompt_ids.empty() ? nullptr : bt->prompt_ids.data(), y)) return -1;
        std::vector<std::vector<int>> pr(B, bt->aed_prompt);
        std::vector<int> caps(B);
        for (int b = 0; b < B; b++) caps[b] = lens[b] + bt->aed_delta;
        std::vector<int> idx;
        for (int b = 0; b < B; b++) if (lens[b] > 0) idx.push_back(b);
        if ((int)idx.size() == B) {
            if (m.decode_aed(y, lens, pr, bt->aed_eos, caps, bt->tokens)) return -1;
        } else {                           // utterances without a single encoder frame produce nothing
            std::vector<int> l2, c2;
            std::vector<std::vector<int>> p2, t2;
            for (int b : idx) { l2.push_back(lens[b]); c2.push_back(caps[b]); p2.push_back(pr[b]); }
            if (!idx.empty() && m.decode_aed(y, l2, p2, bt->aed_eos, c2, t2)) return -1;
            for (size_t i = 0; i < idx.size(); i++) bt->tokens[idx[i]] = t2[i];
        }
        for (int b = 0; b < B; b++) bt->frames[b].assign(bt->tokens[b].size(), 0);
    } else {
        if (m.encoder_post(x, lens, bt->prompt_ids.empty() ? nullptr : bt->prompt_ids.data(), y)) return -1;
        if (m.decode_greedy(y, lens, bt->tokens, bt->frames)) return -1;
    }
    return m.check_status("batch_run");
}

int mynah_b200_batch_run(mynah_b200_model *h, mynah_b200_batch *bt, int decoder) {
    if (!h || !bt) { set_error("batch_run: bad argument"); return -1; }
    Lease lease(h);
    return run_batch_locked(lease.model(), bt, bt->audio.data(), nullptr, decoder);
}

int mynah_b200_batch_fetch(mynah_b200_model *h, mynah_b200_batch *bt, int **tokens, int **frames, int *n_tokens) {
    (void)h;
    if (!bt || (int)bt->tokens.size() != bt->batch) { set_error("batch_fetch: nothing to fetch"); return -1; }
    for (int b = 0; b < bt->batch; b++) {
        const size_t n = bt->tokens[b].size();
        n_tokens[b] = (int)n;
        tokens[b] = (int *)malloc((n ? n : 1) * sizeof(int));
        if (!tokens[b]) { set_error("out of host memory"); return -1; }
        memcpy(tokens[b], bt->tokens[b].data(), n * sizeof(int));
        if (frames) {
            frames[b] = (int *)malloc((n ? n : 1) * sizeof(int));
            if (!frames[b]) { set_error("out of host memory"); return -1; }
            memcpy(frames[b], bt->frames[b].data(), n * sizeof(int));
        }
    }
    return 0;
}

int mynah_b200_transcribe_batch(mynah_b200_model *h, const float *const *audio, const size_t *n_samples, int batch,
                                int decoder, int **tokens, int **frames, int *n_tokens) {
    return mynah_b200_transcribe_batch_prompts(h, audio, n_samples, batch, nullptr, decoder, tokens, frames, n_tokens);
}

int mynah_b200_transcribe_batch_prompts(mynah_b200_model *h, const float *const *audio, const size_t *n_samples, int batch,
                                        const int *prompt_ids, int decoder, int **tokens, int **frames, int *n_tokens) {
    if (!h || !h->m.finalized || batch <= 0 || !audio || !n_samples) { set_error("transcribe_batch: bad argument"); return -1; }
    mynah_b200_batch bt;
    bt.batch = batch;
    bt.n_samples.assign(n_samples, n_samples + batch);
    mynah_b200_batch_set_prompts(&bt, prompt_ids);
    int rc;
    {
        Lease lease(h);
        rc = run_batch_locked(lease.model(), &bt, nullptr, audio, decoder);
        if (rc == 0) lease.idle();
    }
    if (rc == 0) rc = mynah_b200_batch_fetch(h, &bt, tokens, frames, n_tokens);
    return rc;
}

int mynah_b200_transcribe_batch_aed(mynah_b200_model *h, const float *const *audio, const size_t *n_samples, int batch,
                                    const int *prompt, int n_prompt, int eos, int max_gen_delta, int **tokens, int *n_tokens) {
    if (!h || !h->m.finalized || batch <= 0 || !audio || !n_samples || !prompt || n_prompt <= 0) { set_error("transcribe_batch_aed: bad argument"); return -1; }
    mynah_b200_batch bt;
    bt.batch = batch;
    bt.n_samples.assign(n_samples, n_samples + batch);
    mynah_b200_batch_set_aed(&bt, prompt, n_prompt, eos, max_gen_delta);
    int rc;
    {
        Lease lease(h);
        rc = run_batch_locked(lease.model(), &bt, nullptr, audio, 2);
        if (rc == 0) lease.idle();
    }
    if (rc == 0) rc = mynah_b200_batch_fetch(h, &bt, tokens, nullptr, n_tokens);
    return rc;
}

// ------------------------------------------------------------------- qmat API
mynah_b200_qmat *mynah_b200_qmat_create(int fmt, const void *data, const float *scales, int n, int k) {
    if (!mynah_b200_available()) { set_error("no sm_100 CUDA device available"); return nullptr; }
    const int f = internal_fmt(fmt);
    if (f < 0 || !data || n <= 0 || k <= 0) { set_error("qmat_create: bad argument"); return nullptr; }
    // a throw-away Model supplies the upload/dequant plumbing; ownership moves to the handle
    Model tmp;
    if (cudaStreamCreateWithFlags(&tmp.stream, cudaStreamNonBlocking) != cudaSuccess) { set_error("cudaStreamCreate failed"); return nullptr; }
    mynah_b200_qmat *q = new mynah_b200_qmat();
    const bool planes = (k % 64) == 0;
    tmp.status = q->status = (int *)tmp.dev_alloc(QMAT_BLOCK);
    if (!q->status) { delete q; return nullptr; }
    cudaMemset(q->status, 0, QMAT_HEAD);
    cudaDeviceSynchronize();
    if (tmp.upload_weight(q->w, f, data, scales, n, k, planes, false)) { delete q; return nullptr; }
    cudaDeviceSynchronize();
    if (planes && tmp.check_status("qmat_create")) {
        // a weight value outside the fp16 operand range: the handle keeps the stored blocks (small-T products,
        // dequantisation) and drops the planes, so the many-row tensor-core product refuses instead of
        // returning inf / NaN
        q->w.hi = q->w.lo = nullptr;
    }
    q->owned.swap(tmp.owned);
    q->stream = tmp.stream;
    tmp.stream = nullptr;
    static std::atomic<uint64_t> last_id{0};
    q->id = ++last_id;
    q->device = workspace_pool().handle_made();
    return q;
}

void mynah_b200_qmat_free(mynah_b200_qmat *q) {
    if (!q) return;
    const int device = q->device;
    for (mynah_b200_qmat::Graph &g : q->graphs) if (g.exec) cudaGraphExecDestroy(g.exec);
    for (void *p : q->owned) cudaFree(p);                       // waits for the handle's products
    if (q->stream) cudaStreamDestroy(q->stream);
    pinned_pool().give(q->host);
    delete q;
    workspace_pool().handle_gone(device);
}

// device bytes of temporaries that a product of T rows needs beside its input and output
static size_t qmat_temp_bytes(const QWeight &w, int T, int flags) {
    if (flags & MYNAH_B200_A8)
        return w.fmt == FMT_MYNAH_Q8 && T > 16 && w.k % 128 == 0 ? align_up((size_t)T * w.k, 256) + (size_t)T * 4 : 0;
    if (T <= 16 && w.k <= 8192 && !(flags & MYNAH_B200_FEW_ROWS)) return 0;
    return 2 * align_up((size_t)T * w.k * 2, 256);
}

static int qmat_mul_locked(const mynah_b200_qmat *q, const float *x, float *out, int T, int flags, uint8_t *temp);

int mynah_b200_qmat_mul_device(const mynah_b200_qmat *q, const float *x, float *out, int T, int flags) {
    if (!q || !x || !out || T < 0) { set_error("qmat_mul: bad argument"); return -1; }
    if (T == 0) return 0;
    std::lock_guard<std::mutex> lk(q->mu);
    const size_t bytes = qmat_temp_bytes(q->w, T, flags);
    const bool in_block = bytes <= QMAT_TEMP;
    QmatScratch s(q, in_block ? 0 : bytes);
    if (!in_block && !s.get()) { set_error("qmat_mul: device allocation failed"); return -1; }
    return qmat_mul_locked(q, x, out, T, flags, in_block ? (uint8_t *)q->status + QMAT_TEMP_AT : s.get());
}

static int qmat_mul_locked(const mynah_b200_qmat *q, const float *x, float *out, int T, int flags, uint8_t *temp) {
    const QWeight &w = q->w;
    if (flags & MYNAH_B200_A8) {
        if (w.fmt == FMT_MYNAH_Q8 && T > 16 && w.k % 128 == 0) {
            // many rows: the same integers on the tensor cores (bit-identical to the row-dot kernel below)
            int8_t *qx = (int8_t *)temp;
            float *sx = (float *)(temp + align_up((size_t)T * w.k, 256));
            GemmEpilogue e;
            memset(&e, 0, sizeof(e));
            e.mode = OUT_F32; e.act = ACT_NONE; e.alpha = 1.f; e.out = out; e.ldo = w.n;
            int rc = act_quant_rows(x, qx, sx, T, w.k, q->stream);
            if (rc == 0) rc = gemm_i8(qx, w.k, sx, reinterpret_cast<const int8_t *>(w.raw), w.k, w.scales, e, T, w.n, w.k, q->status, q->stream);
            if (rc == 0) note_launch(2);
            return rc;
        }
        const int rc = qgemv_a8(w, x, out, T, nullptr, nullptr, q->stream);
        if (rc == 0) note_launch(2);
        return rc;
    }
    if (T <= 16 && w.k <= 8192 && !(flags & MYNAH_B200_FEW_ROWS)) {     // QMAT_SMALL_T / QMAT_K_MAX of the reference (src/qmat.c:180-181)
        if (w.tc_q && !(flags & (MYNAH_B200_SCALAR | MYNAH_B200_MMA_SYNC))) {
            int rc = 0;
            for (int t0 = 0; t0 < T && rc == 0; t0 += 8)
                rc = qstream_tc(w, x + (size_t)t0 * w.k, w.k, out + (size_t)t0 * w.n, w.n, nullptr, T - t0 < 8 ? T - t0 : 8,
                                q->status, q->stream);
            if (rc == 0) note_launch(((T + 7) / 8) * (w.tc_scratch ? 2 : 1));
            return rc;
        }
        if (w.mma_q && !(flags & MYNAH_B200_SCALAR)) {
            const int rc = qgemv_mma(w, x, w.k, out, w.n, nullptr, T, q->stream);
            if (rc == 0) note_launch((T + 3) / 4);
            return rc;
        }
        const int rc = qgemv(w, x, w.k, out, w.n, nullptr, T, q->stream);
        if (rc == 0) note_launch((T + 3) / 4);
        return rc;
    }
    if (!w.hi) { set_error("qmat_mul: the many-row path needs k %% 64 == 0 (k=%d) and weights below the fp16 operand limit 65504", w.k); return -1; }
    __half *hi = (__half *)temp, *lo = (__half *)(temp + align_up((size_t)T * w.k * 2, 256));
    int rc = split_to_h16(x, hi, lo, (size_t)T * w.k, q->stream, q->status);
    GemmEpilogue e;
    memset(&e, 0, sizeof(e));
    e.mode = OUT_F32; e.act = ACT_NONE; e.alpha = 1.f; e.out = out; e.ldo = w.n;
    GemmOperand A{hi, lo, w.k}, B{w.hi, w.lo, w.k};
    if (rc == 0) rc = (flags & MYNAH_B200_FEW_ROWS) ? gemm_skinny(A, B, e, T, w.n, w.k, (flags & MYNAH_B200_FAST) ? 1 : 3, q->status, q->stream)
                                                    : gemm_tc(A, B, e, T, w.n, w.k, (flags & MYNAH_B200_FAST) ? 1 : 3, q->status, q->stream);
    if (rc == 0) note_launch(2);
    return rc;
}

static int qmat_status(const mynah_b200_qmat *q, int st) {
    if (st == 0) return 0;
    if (st == ST_RANGE) set_error("qmat: a value reached the fp16 operand range (|v| >= 65504) or was not finite");
    else set_error("qmat: a bounded wait inside the contraction kernel ran out (code %d)", st);
    cudaMemsetAsync(q->status, 0, sizeof(int), q->stream);
    cudaStreamSynchronize(q->stream);
    return -1;
}

int mynah_b200_qmat_sync(const mynah_b200_qmat *q) {
    if (!q) { set_error("qmat_sync: null handle"); return -1; }
    int st = 0;
    MB_CUDA(cudaMemcpyAsync(&st, q->status, sizeof(int), cudaMemcpyDeviceToHost, q->stream));
    MB_CUDA(cudaStreamSynchronize(q->stream));
    return qmat_status(q, st);
}

int mynah_b200_qmat_mul(const mynah_b200_qmat *q, const float *x, float *out, int T, int flags) {
    if (!q || !x || !out || T < 0) { set_error("qmat_mul: bad argument"); return -1; }
    if (T == 0) return 0;
    std::lock_guard<std::mutex> lk(q->mu);
    PinnedTwin twin(q);
    uint8_t *host = twin.get();
    if (!host) { set_error("qmat_mul: host allocation failed"); return -1; }
    const size_t nx = (size_t)T * q->w.k * 4, no = (size_t)T * q->w.n * 4;
    uint8_t *block = (uint8_t *)q->status;
    const bool small_x = nx <= QMAT_SMALL, small_out = no <= QMAT_SMALL;
    // small rows and their temporaries (their planes take as much as they do) have a place in the handle's block
    const size_t nt = small_x ? 0 : align_up(qmat_temp_bytes(q->w, T, flags), 256), nxw = small_x ? 0 : align_up(nx, 256);
    const size_t shared = nt + nxw + (small_out ? 0 : no);
    QmatScratch s(q, shared);
    if (shared && !s.get()) { set_error("qmat_mul: device allocation failed"); return -1; }
    float *xd = (float *)(small_x ? block + QMAT_HEAD + QMAT_SMALL : s.get() + nt);
    float *od = (float *)(small_out ? block + QMAT_HEAD : s.get() + nt + nxw);
    uint8_t *temp = small_x ? block + QMAT_TEMP_AT : s.get();
    const void *src = x;
    if (small_x) src = memcpy(host + QMAT_HEAD + QMAT_SMALL, x, nx);
    auto issue = [&]() -> int {
        if (copy_in(xd, src, nx, q->stream)) return -1;
        if (qmat_mul_locked(q, xd, od, T, flags, temp)) return -1;
        const bool ok = cudaMemcpyAsync(host, block, QMAT_HEAD + (small_out ? no : 0), cudaMemcpyDeviceToHost, q->stream) == cudaSuccess;
        if (!small_out && copy_out(out, od, no, q->stream)) return -1;
        if (!ok) { cudaGetLastError(); set_error("qmat_mul: D2H copy failed"); return -1; }
        return 0;
    };
    mynah_b200_qmat::Graph *g = nullptr;
    if (small_x && small_out && !(flags & MYNAH_B200_A8)) {      // (the int8-row path allocates for itself)
        for (auto &e : q->graphs) if (e.uses && e.T == T && e.flags == flags) g = &e;
        if (!g) {
            g = &q->graphs[q->graph_next];
            q->graph_next = (q->graph_next + 1) & 3;
            if (g->exec) cudaGraphExecDestroy(g->exec);
            *g = mynah_b200_qmat::Graph();
            g->T = T; g->flags = flags;
        }
        if (++g->uses == 2) {
            LaunchRecord record;
            cudaGraph_t rec = nullptr;
            if (cudaStreamBeginCapture(q->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
                const int rc = issue();
                const cudaError_t e = cudaStreamEndCapture(q->stream, &rec);
                g->launches = record.launches;
                if (rc || e != cudaSuccess || !rec || cudaGraphInstantiate(&g->exec, rec, 0) != cudaSuccess) g->exec = nullptr;
                if (g->exec) twin.keep();
                if (rec) cudaGraphDestroy(rec);
            }
            cudaGetLastError();
        }
    }
    int rc;
    if (g && g->exec) {
        rc = cudaGraphLaunch(g->exec, q->stream) == cudaSuccess ? 0 : -1;
        if (rc) { cudaGetLastError(); set_error("qmat_mul: graph launch failed"); }
        else note_launch(g->launches);
    } else {
        rc = issue();
    }
    if (cudaStreamSynchronize(q->stream) != cudaSuccess) { cudaGetLastError(); set_error("qmat_mul: a copy or kernel failed"); return -1; }
    if (rc) return rc;
    if (qmat_status(q, *(const int *)host)) return -1;
    if (small_out) memcpy(out, host + QMAT_HEAD, no);
    return 0;
}

int mynah_b200_qmat_block_dots(const mynah_b200_qmat *q, const float *x, int T, int32_t *dots, float *sx, float *out) {
    if (!q || !x || T <= 0) { set_error("qmat_block_dots: bad argument"); return -1; }
    const QWeight &w = q->w;
    const size_t nd = (size_t)T * w.n * (w.k / 32);
    float *xd = nullptr, *od = nullptr, *sd = nullptr;
    int32_t *dd = nullptr;
    if (cudaMalloc(&xd, (size_t)T * w.k * 4) != cudaSuccess || cudaMalloc(&od, (size_t)T * w.n * 4) != cudaSuccess ||
        cudaMalloc(&sd, (size_t)T * 4) != cudaSuccess || cudaMalloc(&dd, nd * 4) != cudaSuccess ||
        cudaMemcpyAsync(xd, x, (size_t)T * w.k * 4, cudaMemcpyHostToDevice, q->stream) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(xd); cudaFree(od); cudaFree(sd); cudaFree(dd);
        set_error("qmat_block_dots: device allocation or copy failed");
        return -1;
    }
    int rc = qgemv_a8(w, xd, od, T, dd, sd, q->stream);
    if (rc == 0) note_launch(2);
    cudaStreamSynchronize(q->stream);
    if (rc == 0 && dots) cudaMemcpy(dots, dd, nd * 4, cudaMemcpyDeviceToHost);
    if (rc == 0 && sx) cudaMemcpy(sx, sd, (size_t)T * 4, cudaMemcpyDeviceToHost);
    if (rc == 0 && out) cudaMemcpy(out, od, (size_t)T * w.n * 4, cudaMemcpyDeviceToHost);
    cudaFree(xd); cudaFree(od); cudaFree(sd); cudaFree(dd);
    if (rc == 0 && cudaGetLastError() != cudaSuccess) { set_error("qmat_block_dots: device error"); rc = -1; }
    return rc;
}

int mynah_b200_qmat_dequant(const mynah_b200_qmat *q, float *wd) {
    if (!q || !wd) { set_error("qmat_dequant: bad argument"); return -1; }
    const QWeight &w = q->w;
    float *d = nullptr;
    MB_CUDA(cudaMalloc(&d, (size_t)w.n * w.k * 4));
    int rc = dequant_to_f32(w.fmt, w.raw, w.scales, d, w.n, w.k, q->stream);
    if (rc == 0) note_launch();
    cudaStreamSynchronize(q->stream);
    if (rc == 0) cudaMemcpy(wd, d, (size_t)w.n * w.k * 4, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return rc;
}

int mynah_b200_gemm_wt(const float *x, const float *w, float *out, int T, int n, int k) {
    if (!x || !w || !out || T <= 0 || n <= 0 || k <= 0) { set_error("gemm_wt: bad argument"); return -1; }
    mynah_b200_qmat *q = mynah_b200_qmat_create(MYNAH_B200_F32, w, nullptr, n, k);
    if (!q) return -1;
    const int rc = mynah_b200_qmat_mul(q, x, out, T, MYNAH_B200_A16);
    mynah_b200_qmat_free(q);
    return rc;
}

// ---- address-keyed resident weights: the calling convention of the reference's own CUDA hook
// (src/cuda_gemm.cu:92-130: every host weight pointer is uploaded once and found again by address).
// One entry per (pointer, format, shape); calls on the same weight take the entry's lock (its
// handle owns one stream and one scratch area), calls on different weights run side by side.
namespace {
// Entries are reference-counted: a call keeps its entry alive while it runs even if another thread
// evicts the cache meanwhile (the device memory goes when the last user lets go).
struct ResidentWeight {
    const void *host; int fmt, n, k;
    mynah_b200_qmat *q;
    std::mutex mu;
    ResidentWeight(const void *h, int f, int n_, int k_, mynah_b200_qmat *q_) : host(h), fmt(f), n(n_), k(k_), q(q_) {}
    ~ResidentWeight() { mynah_b200_qmat_free(q); }
};
std::mutex g_resident_mu;
std::vector<std::shared_ptr<ResidentWeight>> g_resident;

std::shared_ptr<ResidentWeight> resident_lookup(const void *host, int fmt, int n, int k) {
    for (auto &e : g_resident)
        if (e->host == host && e->fmt == fmt && e->n == n && e->k == k) return e;
    return nullptr;
}

std::shared_ptr<ResidentWeight> resident_weight(const void *host, int fmt, const float *scales, int n, int k) {
    {
        std::lock_guard<std::mutex> lk(g_resident_mu);
        if (auto e = resident_lookup(host, fmt, n, k)) return e;
    }
    // upload and re-tile outside the lock: first-touch calls on different weights run side by side
    mynah_b200_qmat *q = mynah_b200_qmat_create(fmt, host, scales, n, k);
    if (!q) return nullptr;
    auto fresh = std::make_shared<ResidentWeight>(host, fmt, n, k, q);
    std::lock_guard<std::mutex> lk(g_resident_mu);
    if (auto e = resident_lookup(host, fmt, n, k)) return e;      // another thread was first; ours is dropped
    g_resident.push_back(fresh);
    return fresh;
}
}  // namespace

int mynah_b200_qgemm(const void *wq, int fmt, const float *scales, int n, int k, const float *x, float *out, int T, int flags) {
    if (!wq || !x || !out || T < 0 || n <= 0 || k <= 0) { set_error("qgemm: bad argument"); return -1; }
    if (!mynah_b200_available()) { set_error("qgemm: no sm_100 device"); return -1; }
    std::shared_ptr<ResidentWeight> e = resident_weight(wq, fmt, scales, n, k);
    if (!e) return -1;
    std::lock_guard<std::mutex> lk(e->mu);
    return mynah_b200_qmat_mul(e->q, x, out, T, flags);
}

void mynah_b200_weights_evict(void) {
    std::vector<std::shared_ptr<ResidentWeight>> drop;
    {
        std::lock_guard<std::mutex> lk(g_resident_mu);
        drop.swap(g_resident);
    }
    // entries still in use by a running call are freed when that call returns
}

int mynah_b200_weights_resident(void) {
    std::lock_guard<std::mutex> lk(g_resident_mu);
    return (int)g_resident.size();
}

// the two symbols src/backend.c:23-26 declares and src/cuda_gemm.cu defines, same meaning:
// 1 / 0, and 0 = done, -1 = the caller falls back
int mynah_asr_cuda_available(void) { return mynah_b200_available(); }

int mynah_asr_cuda_gemm_wt(const float *x, const float *w, float *out, int T, int n, int k) {
    return mynah_b200_qgemm(w, MYNAH_B200_F32, nullptr, n, k, x, out, T, MYNAH_B200_A16);
}

void mynah_b200_profile_begin(mynah_b200_model *h) {
    if (!h) return;
    Lease lease(h, 0);      // the first context: the one a single-threaded caller always runs on
    Model &m = lease.model();
    m.prof_on = true; m.prof_used = 0;
    for (int i = 0; i < Model::PROF_NCAT; i++) { m.prof_flops[i] = 0; m.prof_bytes[i] = 0; m.prof_launches[i] = 0; }
}

int mynah_b200_profile_end(mynah_b200_model *h, double *ms, double *flops, long long *launches, int ncat) {
    if (!h) { set_error("profile_end: null model"); return -1; }
    Lease lease(h, 0);      // the first context: the one a single-threaded caller always runs on
    Model &m = lease.model();
    m.prof_on = false;
    MB_CUDA(cudaStreamSynchronize(m.stream));
    for (int i = 0; i < ncat; i++) { ms[i] = 0; flops[i] = 0; launches[i] = 0; }
    for (size_t i = 0; i < m.prof_used; i++) {
        float t = 0.f;
        if (cudaEventElapsedTime(&t, m.prof_spans[i].a, m.prof_spans[i].b) == cudaSuccess && m.prof_spans[i].cat < ncat)
            ms[m.prof_spans[i].cat] += t;
    }
    for (int i = 0; i < ncat && i < Model::PROF_NCAT; i++) { flops[i] = m.prof_flops[i]; launches[i] = m.prof_launches[i]; }
    m.prof_used = 0;
    return 0;
}

void mynah_b200_profile_bytes(mynah_b200_model *h, double *bytes, int ncat) {
    for (int i = 0; i < ncat; i++) bytes[i] = (h && i < Model::PROF_NCAT) ? h->m.prof_bytes[i] : 0.0;
}

void mynah_b200_decoder_clocks(mynah_b200_model *h, long long *out8) {
    for (int i = 0; i < 8; i++) out8[i] = h ? h->m.dec_dbg[i] : 0;
}

int mynah_b200_sigmoid(const float *x, float *out, int n, int cell) {
    if (!x || !out || n <= 0) { set_error("sigmoid: bad argument"); return -1; }
    float *d = nullptr;
    MB_CUDA(cudaMalloc(&d, (size_t)n * 4));
    int rc = cudaMemcpy(d, x, (size_t)n * 4, cudaMemcpyHostToDevice) == cudaSuccess ? sigmoids(d, d, n, cell, nullptr) : -1;
    if (rc == 0) note_launch();
    if (rc == 0 && cudaMemcpy(out, d, (size_t)n * 4, cudaMemcpyDeviceToHost) != cudaSuccess) rc = -1;
    if (rc) { cudaGetLastError(); set_error("sigmoid: a copy or kernel failed"); }
    cudaFree(d);
    return rc;
}

double mynah_b200_qmat_time(const mynah_b200_qmat *q, int T, int flags, int iters) {
    if (!q || T <= 0 || iters <= 0) { set_error("qmat_time: bad argument"); return -1.0; }
    const QWeight &w = q->w;
    float *x = nullptr, *out = nullptr;
    __half *hi = nullptr, *lo = nullptr;
    if (cudaMalloc(&x, (size_t)T * w.k * 4) != cudaSuccess || cudaMalloc(&out, (size_t)T * w.n * 4) != cudaSuccess) { set_error("qmat_time: cudaMalloc failed"); return -1.0; }
    cudaMemset(x, 0, (size_t)T * w.k * 4);
    cudaDeviceSynchronize();
    const bool i8 = (flags & MYNAH_B200_A8) && w.fmt == FMT_MYNAH_Q8 && T > 16 && w.k % 128 == 0;
    int8_t *qx = nullptr;
    float *sx = nullptr;
    if (i8) {          // the integer contraction alone: rows quantised once, outside the timed launches
        if (cudaMalloc((void **)&qx, (size_t)T * w.k) != cudaSuccess || cudaMalloc((void **)&sx, (size_t)T * 4) != cudaSuccess ||
            act_quant_rows(x, qx, sx, T, w.k, q->stream)) { cudaFree(x); cudaFree(out); cudaFree(qx); cudaFree(sx); set_error("qmat_time: setup failed"); return -1.0; }
    }
    const bool small = !i8 && !(flags & MYNAH_B200_FEW_ROWS) && ((T <= 16 && w.k <= 8192) || (flags & MYNAH_B200_A8));
    if (!small && !i8) {
        if (!w.hi) { set_error("qmat_time: no operand planes"); cudaFree(x); cudaFree(out); return -1.0; }
        cudaMalloc(&hi, (size_t)T * w.k * 2); cudaMalloc(&lo, (size_t)T * w.k * 2);
        split_to_h16(x, hi, lo, (size_t)T * w.k, q->stream);
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0); cudaEventCreate(&e1);
    int rc = 0;
    for (int it = -2; it < iters && rc == 0; it++) {
        if (it == 0) cudaEventRecord(e0, q->stream);
        if (i8) {
            GemmEpilogue e;
            memset(&e, 0, sizeof(e));
            e.mode = OUT_F32; e.alpha = 1.f; e.out = out; e.ldo = w.n;
            rc = gemm_i8(qx, w.k, sx, reinterpret_cast<const int8_t *>(w.raw), w.k, w.scales, e, T, w.n, w.k, q->status, q->stream);
        } else if (small) rc = (flags & MYNAH_B200_A8) ? qgemv_a8(w, x, out, T, nullptr, nullptr, q->stream)
                   : (w.tc_q && T <= 8 && !(flags & (MYNAH_B200_SCALAR | MYNAH_B200_MMA_SYNC))) ? qstream_tc(w, x, w.k, out, w.n, nullptr, T, q->status, q->stream)
                   : (w.mma_q && !(flags & MYNAH_B200_SCALAR)) ? qgemv_mma(w, x, w.k, out, w.n, nullptr, T, q->stream)
                   : qgemv(w, x, w.k, out, w.n, nullptr, T, q->stream);
        else {
            GemmEpilogue e;
            memset(&e, 0, sizeof(e));
            e.mode = OUT_F32; e.alpha = 1.f; e.out = out; e.ldo = w.n;
            GemmOperand A{hi, lo, w.k}, B{w.hi, w.lo, w.k};
            rc = (flags & MYNAH_B200_FEW_ROWS) ? gemm_skinny(A, B, e, T, w.n, w.k, (flags & MYNAH_B200_FAST) ? 1 : 3, q->status, q->stream)
                                               : gemm_tc(A, B, e, T, w.n, w.k, (flags & MYNAH_B200_FAST) ? 1 : 3, q->status, q->stream);
        }
        if (it >= 0) note_launch();
    }
    cudaEventRecord(e1, q->stream);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0); cudaEventDestroy(e1);
    cudaFree(x); cudaFree(out); if (hi) cudaFree(hi); if (lo) cudaFree(lo); if (qx) cudaFree(qx); if (sx) cudaFree(sx);
    if (rc != 0 || cudaGetLastError() != cudaSuccess) { if (rc == 0) set_error("qmat_time: device error"); return -1.0; }
    return (double)ms / iters;
}

}  // extern "C"
