// Host side of the C ABI (include/es_gb300.h): validates a plan descriptor, derives every
// device table in C++ (the production cascade's in es_cascade.cu; for counting and scalar launches
// sorted inner ring, carry-split keys and buckets, ring-1 residue table, ring-2 delta table and
// word-mask phase tables), uploads a table set when a launch first needs it, and drives
// single-plan launches (the reference GpuSieve._launch surface) and persistent batch launches
// with CUDA-graph replay.  No exception crosses the ABI: every entry point returns an int.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <exception>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/es_gb300.h"
#include "es_cascade.h"
#include "es_internal.h"

typedef es_u128 u128;

namespace {

thread_local std::string g_err;

int fail(int code, const std::string& msg) {
    g_err = msg;
    return code;
}

int cuda_fail(cudaError_t e, const char* what) {
    g_err = std::string(what) + ": " + cudaGetErrorString(e);
    return ES_ERR_CUDA;
}

// The end of an entry point that allocates on the host: nothing throws across the ABI.
#define ES_CATCH                                                                     \
    catch (const std::exception&) { return fail(ES_ERR_NOMEM, "host allocation"); }

#define ES_CUDA(call, what)                                  \
    do {                                                     \
        cudaError_t _e = (call);                             \
        if (_e != cudaSuccess) return cuda_fail(_e, what);   \
    } while (0)

struct DeviceFacts {
    int dev = -1;
    int sms = 0;
    int smem_optin = 0;
    bool prepared = false;
};
DeviceFacts g_dev;

int device_facts() {
    int dev = 0;
    ES_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    if (g_dev.dev == dev && g_dev.prepared) return ES_OK;
    int major = 0, minor = 0;
    ES_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev), "attr");
    ES_CUDA(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev), "attr");
    if (major != 10 || minor != 3)
        return fail(ES_ERR_NODEV, "device is sm_" + std::to_string(major * 10 + minor) +
                                      ", this library is built for sm_103a only");
    g_dev.dev = dev;
    ES_CUDA(cudaDeviceGetAttribute(&g_dev.sms, cudaDevAttrMultiProcessorCount, dev), "attr");
    ES_CUDA(cudaDeviceGetAttribute(&g_dev.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev),
            "attr");
    int e = es_scan_prepare(g_dev.smem_optin - 1024);
    if (e) return cuda_fail((cudaError_t)e, "cudaFuncSetAttribute(scan)");
    g_dev.prepared = true;
    return ES_OK;
}

int check_tune(const es_tune& t) {
    if (t.layout > ES_LAYOUT_AUTO)
        return fail(ES_ERR_ARG, "tune.layout must be 0 (word-mask), 1 (scalar), 2 (pair), 3 (word masks in shared "
                                "memory), 4 (pair tables in shared memory) or 5 (chosen per launch)");
    if (t.mask_filters < 1 || t.mask_filters > ES_MAX_MASK_FILTERS)
        return fail(ES_ERR_ARG, "tune.mask_filters must be in 1..8");
    if (t.threads < 64 || t.threads > 1024 || t.threads % 32)
        return fail(ES_ERR_ARG, "tune.threads must be a multiple of 32 in [64, 1024]");
    if (t.strip < 1 || t.strip > 4096) return fail(ES_ERR_ARG, "tune.strip must be in 1..4096");
    if (t.ctas_per_sm < 1 || t.ctas_per_sm > 16)
        return fail(ES_ERR_ARG, "tune.ctas_per_sm must be in 1..16");
    return ES_OK;
}

es_tune default_tune() {
    es_tune t;
    t.layout = ES_LAYOUT_WORDMASK;
    t.mask_filters = 4;
    t.threads = 512;
    t.strip = 8;
    t.smem_kb = 0;
    t.ctas_per_sm = 4;
    t.count_stages = 0;
    t.reserved = 0;
    return t;
}

}  // namespace

// ------------------------------------------------------------------------------------------
namespace {

// One set of device tables of a plan: the header and its arena.
struct TableSet {
    EsInst h{};
    EsInst* d = nullptr;
    unsigned char* arena = nullptr;
    uint64_t bytes = 0;
};

struct ProdSet {
    TableSet t;
    std::vector<EsCascadeEntry> entries;
};

// Device and pinned memory, stream and events of one batch.  A destroyed batch hands them to its
// device's pool for the next batch: a block-ordered search makes a batch per launch, and allocating
// and freeing these took 200 of its 254 us.
struct BatchMem {
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    unsigned char *dev = nullptr, *pin = nullptr;
    size_t dev_cap = 0, pin_cap = 0;
    es_survivor* surv = nullptr;
    uint64_t surv_cap = 0;
    BatchMem() = default;
    BatchMem(const BatchMem&) = delete;
    BatchMem& operator=(const BatchMem&) = delete;
    size_t bytes() const { return dev_cap + pin_cap + sizeof(es_survivor) * surv_cap; }
    ~BatchMem() {
        cudaFree(dev);
        cudaFree(surv);
        if (pin) cudaFreeHost(pin);
        if (ev0) cudaEventDestroy(ev0);
        if (ev1) cudaEventDestroy(ev1);
        if (stream) cudaStreamDestroy(stream);
    }
    cudaError_t need(size_t dev_bytes, size_t pin_bytes, uint64_t cap) {
        cudaError_t e = cudaSuccess;
        if (!stream) e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
        if (e == cudaSuccess && !ev0) e = cudaEventCreate(&ev0);
        if (e == cudaSuccess && !ev1) e = cudaEventCreate(&ev1);
        if (e == cudaSuccess && dev_cap < dev_bytes) {
            cudaFree(dev);
            dev = nullptr;
            dev_cap = 0;
            e = cudaMalloc(&dev, dev_bytes * 2);
            if (e == cudaSuccess) dev_cap = dev_bytes * 2;
        }
        if (e == cudaSuccess && pin_cap < pin_bytes) {
            if (pin) cudaFreeHost(pin);
            pin = nullptr;
            pin_cap = 0;
            e = cudaHostAlloc(&pin, pin_bytes * 2, cudaHostAllocDefault);
            if (e == cudaSuccess) pin_cap = pin_bytes * 2;
        }
        if (e == cudaSuccess && surv_cap < cap) {
            cudaFree(surv);
            surv = nullptr;
            surv_cap = 0;
            e = cudaMalloc(&surv, sizeof(es_survivor) * cap);
            if (e == cudaSuccess) surv_cap = cap;
        }
        return e;
    }
};

// One per device, held by its contexts and their batches and gone with the last of them.
struct BatchPool {
    static constexpr size_t kKeep = 256u << 20;   // idle bytes at most; what is beyond is freed
    std::mutex mu;
    std::vector<std::unique_ptr<BatchMem>> idle;
    // a set whose survivor buffer holds `cap` records, if there is one, else any
    std::unique_ptr<BatchMem> take(uint64_t cap) {
        std::lock_guard<std::mutex> lock(mu);
        if (idle.empty()) return nullptr;
        size_t at = idle.size() - 1;
        for (size_t i = 0; i < idle.size(); ++i)
            if (idle[i]->surv_cap >= cap) at = i;
        std::unique_ptr<BatchMem> m = std::move(idle[at]);
        idle.erase(idle.begin() + (ptrdiff_t)at);
        return m;
    }
    void give(std::unique_ptr<BatchMem> m) {
        std::lock_guard<std::mutex> lock(mu);
        size_t bytes = m->bytes();
        for (const std::unique_ptr<BatchMem>& x : idle) bytes += x->bytes();
        if (bytes > kKeep) return;
        try {
            idle.push_back(std::move(m));
        } catch (const std::exception&) {   // no memory for the list: the set is freed
        }
    }
    static std::shared_ptr<BatchPool> of_device(int dev) {
        static std::mutex mu;
        static std::map<int, std::weak_ptr<BatchPool>> pools;
        std::lock_guard<std::mutex> lock(mu);
        std::shared_ptr<BatchPool> p = pools[dev].lock();
        if (!p) pools[dev] = p = std::make_shared<BatchPool>();
        return p;
    }
};

}  // namespace

struct es_ctx {
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    es_tune tune{};
    EsHostPlan plan;
    EsInst geo{};                 // geometry only (rings, filter count, M)
    TableSet caller;              // caller's cascade order: counting and scalar launches
    ProdSet prod[ES_PMAX + 1];    // production cascade by inner tables
    uint32_t own_tables[ES_PMAX + 1] = {0};   // by tables asked for: tables of this plan's own launches
    std::vector<uint32_t> q;
    u128 M = 1;
    uint32_t tconst[ES_MAX_FILTERS] = {0};
    uint64_t t = 0;
    // launch state
    unsigned long long* d_counts = nullptr;
    es_survivor* d_surv = nullptr;
    uint64_t surv_cap = 0;
    unsigned long long* d_surv_n = nullptr;
    unsigned long long* d_unit = nullptr;   // work counter, and CTAs done: 0 between launches
    unsigned long long* d_done = nullptr;
    unsigned long long* d_min = nullptr;
    unsigned long long* h_pin = nullptr;  // pinned scalars for small readbacks
    uint64_t* d_list = nullptr;
    uint64_t list_cap = 0;
    // the survivor count read since the last launch or reset, if any
    bool count_known = false;
    uint64_t count = 0;
    std::shared_ptr<BatchPool> pool;   // the device's
};

struct es_batch {
    std::shared_ptr<BatchPool> pool;
    std::unique_ptr<BatchMem> mem;
    cudaStream_t stream = nullptr;        // mem's
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    es_tune tune{};
    std::vector<es_ctx*> ctxs;
    std::vector<EsItem> h_items;
    uint32_t n_groups = 0;
    EsItem* d_items = nullptr;
    EsItem* d_items_launch = nullptr;  // the items grouped by width class, as the launches see them
    uint32_t* d_tconst = nullptr;
    std::vector<uint64_t> count_off;
    es_survivor* d_surv = nullptr;
    uint64_t surv_cap = 0;
    // one block of scalars: the group minima and the survivor count (copied to h_result at the end
    // of a run), then the launches' unit counters, the items' and the stage counts; then found
    unsigned long long* d_min = nullptr;         // [n_groups][4]
    unsigned long long* d_surv_n = nullptr;
    unsigned long long* d_unit = nullptr;        // [n_items], one per launch
    unsigned long long* d_item_next = nullptr;   // [n_items] next warp-unit (several plans)
    unsigned long long* d_counts = nullptr;
    unsigned long long* d_found = nullptr;       // [n_groups]
    size_t zero_bytes = 0;                       // from d_surv_n up to d_found
    unsigned long long* h_result = nullptr;      // pinned: minima, count
    uint32_t n_items = 0;
    // One persistent launch per inner-ring width class (1, 2, 3-4 words, wider): each runs the
    // kernel instance specialised for its width instead of one generic instance for all.
    struct Sub {
        EsLaunch L{};
        int grid = 0;
        uint32_t words = 0;
        uint32_t layout = 0;   // the layout this launch runs (launch_layout)
    };
    std::vector<Sub> subs;
    bool ran = false;
};

namespace {

// Shared-memory plan of one launch:
// [small tables | staged phase tables (ES_LAYOUT_SMEM, _SMEM_PAIR) | per-warp stage counters |
//  per-warp slots].
struct SmemPlan {
    uint32_t stage_off, cnt_off, queue_off, bytes;
};

// per-warp slot: entry queue, lane records, tail context (the kernel's EsQueue)
constexpr uint32_t kQueueBytes = ES_QUEUE_BYTES;

SmemPlan plan_smem(uint32_t small_max, uint32_t nf_max, const es_tune& tune, uint32_t stage_words = 0) {
    SmemPlan p;
    const uint32_t warps = tune.threads / 32u;
    const uint32_t queues = kQueueBytes * warps;
    // per-warp stage counters exist only in counting launches; shared memory is kept small so
    // that the CUDA driver's carveout leaves the rest of the SM's 256 KB to L1 (the phase tables),
    // unless the launch stages those tables in shared memory itself
    const uint32_t counters = tune.count_stages ? (uint32_t)es_align_up(4ull * nf_max * warps, 16) : 0u;
    p.stage_off = small_max;
    p.cnt_off = p.stage_off + (uint32_t)es_align_up(4ull * stage_words, 16);
    p.queue_off = p.cnt_off + counters;
    p.bytes = p.queue_off + queues;
    return p;
}

// Words of inner-stage tables a launch of `layout` copies into shared memory, given the word-mask
// words of its first F filters (EsInst::mask_off[F]): those words (ES_LAYOUT_SMEM), twice them as
// pair tables (ES_LAYOUT_SMEM_PAIR), or none.
uint32_t staged_words(uint32_t layout, uint32_t mask_words) {
    if (layout == ES_LAYOUT_SMEM) return mask_words;
    if (layout == ES_LAYOUT_SMEM_PAIR) return 2u * mask_words;
    return 0u;
}

// Word-mask bytes of the inner-stage tables that fit the L1 beside the scan's own shared memory.
constexpr uint32_t kL1TableBudget = 180u * 1024u;

// The layout a launch actually runs, given the word-mask words of its inner-stage tables (the
// largest among its plans).  A staged layout only for inner rings of one or two words whose
// staged tables fit the opt-in shared memory beside the rest of the launch's shared memory;
// otherwise the same tables read through L1 (word masks, or pair tables).  ES_LAYOUT_AUTO: staged
// word masks where they fit, else word masks through L1 when those fit L1 and pair tables would
// not, else pair tables (wider rings: word masks).  No choice changes which candidates pass.
uint32_t launch_layout(uint32_t layout, uint32_t words, uint32_t small_max, uint32_t nf_max,
                       const es_tune& tune, uint32_t mask_words) {
    auto fits = [&](uint32_t l) {
        return plan_smem(small_max, nf_max, tune, staged_words(l, mask_words)).bytes <=
               (uint32_t)g_dev.smem_optin - 1024u;
    };
    const bool narrow = words == 1 || words == 2;
    if (layout == ES_LAYOUT_AUTO) {
        if (!narrow) return ES_LAYOUT_WORDMASK;
        if (fits(ES_LAYOUT_SMEM)) return ES_LAYOUT_SMEM;
        const uint64_t bytes = 4ull * mask_words;
        return (bytes <= kL1TableBudget && kL1TableBudget < 2 * bytes) ? ES_LAYOUT_WORDMASK : ES_LAYOUT_PAIR;
    }
    if (layout != ES_LAYOUT_SMEM && layout != ES_LAYOUT_SMEM_PAIR) return layout;
    if (!narrow) return ES_LAYOUT_WORDMASK;
    if (fits(layout)) return layout;
    return layout == ES_LAYOUT_SMEM ? ES_LAYOUT_WORDMASK : ES_LAYOUT_PAIR;
}

// Filters of the inner-ring stage actually compiled into the launched kernel: word-mask kernels
// are instantiated for exactly 0..6 and 8 filters (never more than the plan has or the tables
// built); the scalar layout takes a runtime count.
uint32_t stage_filters(uint32_t layout, uint32_t requested, uint32_t nf, uint32_t built) {
    if (layout == ES_LAYOUT_SCALAR) return std::max<uint32_t>(requested, 1);
    uint32_t f = std::min(std::min(requested, nf), built);
    return f == 7 ? 6 : f;
}

int grid_for(uint32_t layout, uint32_t count, uint32_t words, uint32_t filters, const es_tune& tune,
             uint32_t smem, uint64_t units, int* grid) {
    int occ = 0;
    int e = es_scan_occupancy((int)layout, (int)count, words, filters, (int)tune.threads,
                              (int)smem, &occ);
    if (e) return cuda_fail((cudaError_t)e, "occupancy");
    if (occ < 1) return fail(ES_ERR_ARG, "launch shape does not fit one SM (threads/smem)");
    uint64_t g = (uint64_t)g_dev.sms * (uint64_t)std::min<uint32_t>((uint32_t)occ, tune.ctas_per_sm);
    if (units < g) g = units;
    if (g < 1) g = 1;
    *grid = (int)g;
    return ES_OK;
}

uint64_t cycles_of(const EsInst& I, uint64_t ob, uint64_t oe, uint64_t* cb) {
    *cb = ob / I.r1;
    const uint64_t ce = (oe + I.r1 - 1) / I.r1;
    return ce - *cb;
}

// Warp-units of the ring-1 cycles [cb, ce) (the kernel's unit decode follows the same rule):
// with a ring 2, 32 ring-2 rows x one window of at most `strip` ring-2 digits (ceil(r2 / strip)
// balanced windows per row); without one, 32 lanes x `strip` consecutive cycles.
uint64_t units_of(const EsInst& I, uint64_t cb, uint64_t ce, uint32_t strip) {
    if (ce <= cb) return 0;
    if (I.r2 <= 1) return (ce - cb + 32ull * strip - 1) / (32ull * strip);
    const uint64_t rows = (ce + I.r2 - 1) / I.r2 - cb / I.r2;
    return (rows + 31) / 32 * ((I.r2 + strip - 1) / strip);
}

// Launches that count no stages run the production cascade, in every layout but the scalar one
// (the layouts are forms of the caller's cascade; none changes which candidates pass).
bool is_production(const es_tune& t) { return !t.count_stages && t.layout != ES_LAYOUT_SCALAR; }

// The shape a production launch runs: the largest CTA that a caller can ask for stands for the
// largest that the production kernel takes.
es_tune prod_shape(es_tune t) {
    if (t.threads == 512)
        t.threads = ES_PROD_THREADS;
    else if (t.threads > 512)
        t.threads = 1024;   // no kernel takes it: the launch is refused
    return t;
}

// Longest unit, in ring-1 cycles per lane, of a plan at `strip` (windows of ring-2 digits are balanced).
uint32_t longest_of(const EsInst& I, uint32_t strip) {
    if (I.r2 <= 1) return strip;
    const uint32_t J = (I.r2 + strip - 1) / strip;
    return (I.r2 + J - 1) / J;
}

// Ring-1 cycles per lane and warp-unit of a launch of `steps` warp-wide cycles, at most the caller's;
// units(s) is the number of units at s, longest(s) the longest of them.  A unit costs about half a
// cycle to set up, so long ones are better; but a warp takes as long for a unit when the SM is half
// empty as when it is full, so a launch of few waves takes whole ones.  Measured when the rule was made
// (3040 resident warps): k = 300, 2^30 positions 103 us in 1.9 waves of 7 cycles, 117 in 4.4 of 3, 141 in 13.3 of 1;
// 2^34 positions 1470 at 7, 1723 at 2; k = 384, 2^28 positions 67 us in 1.5 waves of 1, 127 in 0.2 of 8.
template <class Units, class Longest>
uint32_t launch_strip(uint64_t steps, const es_tune& t, const Units& units, const Longest& longest) {
    const double warps = (double)g_dev.sms * (t.threads / 32u);
    uint32_t best = 1;
    double least = 0.0;
    for (uint32_t s = 1; s <= std::min<uint32_t>(t.strip, 64); ++s) {
        const uint64_t n = units(s);
        if (n == 0) break;
        const double waves = n / warps;
        const double cost = (waves < 8.0 ? std::ceil(waves) : waves + 0.5) *
                            ((waves < 4.0 ? longest(s) : (double)steps / n) + 0.5);
        if (s == 1 || cost < least) {
            least = cost;
            best = s;
        }
    }
    return best;
}

// Warp-wide ring-1 cycles of [cb, ce) (rows of 32 lanes x ring-2 digits).
uint64_t steps_of(const EsInst& I, uint64_t cb, uint64_t ce) {
    if (ce <= cb) return 0;
    if (I.r2 <= 1) return (ce - cb + 31) / 32;
    return ((ce + I.r2 - 1) / I.r2 - cb / I.r2 + 31) / 32 * I.r2;
}

void launch_tables(EsLaunch& L, const EsInst& I) {
    L.small = I.small;
    L.tabs = I.masks;
    L.small_bytes = I.small_bytes;
    L.tab_words = I.tab_words;
}

// Inner tables of a production launch.
uint32_t prod_tables(const es_tune& t) { return std::min<uint32_t>(std::max<uint32_t>(t.mask_filters, 1), ES_PMAX); }

// Whether launches of this shape run the production cascade with PF tables: a plan whose rings are so
// large that the cascade's tables do not fit one CTA runs the scalar layout instead.
bool runs_production(const es_ctx* c, const es_tune& t, uint32_t PF) {
    if (!is_production(t)) return false;
    const EsInst& I = c->prod[PF].t.h;
    return plan_smem(I.small_bytes, I.n_filters, prod_shape(t), I.tab_words).bytes <= (uint32_t)g_dev.smem_optin - 1024u;
}

// The production cascade's block constants from the caller's.
void prod_tconst(const ProdSet& S, const uint32_t* tconst, uint32_t* out) {
    for (size_t i = 0; i < S.entries.size(); ++i) {
        const EsCascadeEntry& e = S.entries[i];
        uint64_t r = 0;
        for (const EsCascadeEntry::Part& p : e.parts) {
            const uint64_t x = tconst[p.f] % p.d;
            r = (r + x * p.unit) % e.q;
        }
        out[i] = (uint32_t)r;
    }
}

// tconst[j] = (t mod q)(M mod q) mod q
void block_tconst(const es_ctx* c, uint64_t t, uint32_t* out) {
    for (size_t f = 0; f < c->q.size(); ++f) {
        const uint64_t q = c->q[f];
        out[f] = (uint32_t)((t % q) * (uint64_t)(c->M % q) % q);
    }
}

}  // namespace

void es_set_last_error(const char* msg) { g_err = msg ? msg : ""; }

// ------------------------------------------------------------------------------------------
extern "C" {

const char* es_last_error(void) { return g_err.c_str(); }

int es_abi_version(void) { return ES_ABI_VERSION; }

int es_device_info(int* sm_count, int* cc_major, int* cc_minor, uint64_t* smem_optin_bytes) {
    int dev = 0;
    ES_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    int a = 0, b = 0, s = 0, o = 0;
    ES_CUDA(cudaDeviceGetAttribute(&a, cudaDevAttrComputeCapabilityMajor, dev), "attr");
    ES_CUDA(cudaDeviceGetAttribute(&b, cudaDevAttrComputeCapabilityMinor, dev), "attr");
    ES_CUDA(cudaDeviceGetAttribute(&s, cudaDevAttrMultiProcessorCount, dev), "attr");
    ES_CUDA(cudaDeviceGetAttribute(&o, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev), "attr");
    if (sm_count) *sm_count = s;
    if (cc_major) *cc_major = a;
    if (cc_minor) *cc_minor = b;
    if (smem_optin_bytes) *smem_optin_bytes = (uint64_t)o;
    return ES_OK;
}

int es_device_name(char* out, uint32_t cap) {
    if (!out || cap == 0) return fail(ES_ERR_ARG, "null or empty output buffer");
    int dev = 0;
    ES_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    cudaDeviceProp prop;
    ES_CUDA(cudaGetDeviceProperties(&prop, dev), "cudaGetDeviceProperties");
    snprintf(out, cap, "%s", prop.name);
    return ES_OK;
}

int es_ctx_destroy(es_ctx* c) {
    if (!c) return ES_OK;
    if (c->stream) cudaStreamSynchronize(c->stream);
    cudaFree(c->caller.arena);
    for (ProdSet& p : c->prod) cudaFree(p.t.arena);
    cudaFree(c->d_counts);
    cudaFree(c->d_surv);
    cudaFree(c->d_surv_n);
    cudaFree(c->d_list);
    if (c->h_pin) cudaFreeHost(c->h_pin);
    if (c->ev0) cudaEventDestroy(c->ev0);
    if (c->ev1) cudaEventDestroy(c->ev1);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
    return ES_OK;
}

// Uploads one table set: the header, the small block, the inner-stage tables and the bit tables
// (ring terms too) in one arena.
static int upload_set(es_ctx* c, TableSet& T, const std::vector<unsigned char>& small, const std::vector<uint32_t>& masks,
                      const std::vector<uint32_t>& pairs, const std::vector<uint32_t>& bits,
                      const std::vector<u128>& terms) {
    const EsHostPlan& P = c->plan;
    size_t aoff = 0;
    auto atake = [&](size_t bytes) { size_t o = aoff; aoff = es_align_up(aoff + bytes, 256); return o; };
    const size_t a_inst = atake(sizeof(EsInst));
    const size_t a_small = atake(small.size());
    const size_t a_masks = atake(4ull * std::max<size_t>(masks.size(), 4));
    const size_t a_pairs = atake(4ull * std::max<size_t>(pairs.size(), 4));
    const size_t a_bits = atake(4ull * std::max<size_t>(bits.size(), 4));
    const size_t a_terms = atake(16ull * std::max<size_t>(terms.size(), 1));
    const size_t a_roff = atake(4ull * P.roff.size());
    const size_t a_radix = atake(4ull * P.radix.size());
    std::vector<unsigned char> img(aoff, 0);
    memcpy(&img[a_small], small.data(), small.size());
    if (!masks.empty()) memcpy(&img[a_masks], masks.data(), 4ull * masks.size());
    if (!pairs.empty()) memcpy(&img[a_pairs], pairs.data(), 4ull * pairs.size());
    if (!bits.empty()) memcpy(&img[a_bits], bits.data(), 4ull * bits.size());
    for (size_t i = 0; i < terms.size(); ++i) {
        uint64_t lo = (uint64_t)terms[i], hi = (uint64_t)(terms[i] >> 64);
        memcpy(&img[a_terms + 16 * i], &lo, 8);
        memcpy(&img[a_terms + 16 * i + 8], &hi, 8);
    }
    memcpy(&img[a_roff], P.roff.data(), 4ull * P.roff.size());
    memcpy(&img[a_radix], P.radix.data(), 4ull * P.radix.size());
    unsigned char* arena = nullptr;
    ES_CUDA(cudaMalloc(&arena, aoff), "cudaMalloc(arena)");
    EsInst& I = T.h;
    I.small = arena + a_small;
    I.masks = reinterpret_cast<const uint32_t*>(arena + a_masks);
    I.pairs = reinterpret_cast<const uint32_t*>(arena + a_pairs);
    I.allowed = reinterpret_cast<const uint32_t*>(arena + a_bits);
    I.ring_terms = reinterpret_cast<const uint64_t*>(arena + a_terms);
    I.ring_off = reinterpret_cast<const uint32_t*>(arena + a_roff);
    I.radix = reinterpret_cast<const uint32_t*>(arena + a_radix);
    memcpy(&img[a_inst], &I, sizeof(EsInst));
    // the copy may still be on its way to the device when it returns, and no stream that reads the
    // tables is ordered after the default stream: wait for it
    cudaError_t ce = cudaMemcpy(arena, img.data(), aoff, cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(nullptr);
    if (ce != cudaSuccess) {
        cudaFree(arena);
        return cuda_fail(ce, "table upload");
    }
    T.arena = arena;
    T.d = reinterpret_cast<EsInst*>(arena + a_inst);
    T.bytes = aoff;
    return ES_OK;
}

// Tables of the caller's cascade order (counting launches and the scalar layout).
static int build_caller(es_ctx* c) {
    const EsHostPlan& P = c->plan;
    TableSet T;
    EsInst& I = T.h;
    I = c->geo;
    const u128 M = P.M;
    const uint32_t r0 = I.r0, r1 = I.r1, r2 = I.r2, W = I.W, nf = I.n_filters, sh = I.sh;
    const uint32_t FB = std::min<uint32_t>(ES_FMAX, nf);
    std::vector<EsFilterC> fc(nf);
    for (uint32_t f = 0; f < nf; ++f) fc[f] = es_filter_consts(M, P.q[f], P.bit_off[f]);
    const EsSortedRing R = es_sort_inner(P);
    const uint32_t kbits = es_bitlen(M >> sh);
    const uint32_t bsh = kbits > ES_NBUCKET_LOG2 ? kbits - ES_NBUCKET_LOG2 : 0;
    std::vector<uint32_t> K0(r0);
    for (uint32_t i = 0; i < r0; ++i) K0[i] = (uint32_t)(R.S0[i] >> sh);
    // bucket b: the first sorted slot whose key is >= b << bsh, and the keys of that slot and
    // the next two (0xffffffff past the end), so that one 16-byte load settles the split
    std::vector<uint32_t> BK(4ull * (ES_NBUCKET + 1));
    for (uint32_t bkt = 0, n = 0; bkt <= ES_NBUCKET; ++bkt) {
        const uint64_t lim = (uint64_t)bkt << bsh;
        while (n < r0 && (uint64_t)K0[n] < lim) ++n;
        BK[4 * bkt] = n;
        for (uint32_t j = 0; j < 3; ++j) BK[4 * bkt + 1 + j] = n + j < r0 ? K0[n + j] : 0xffffffffu;
    }
    // ---- small block ----------------------------------------------------------------------
    EsSmallBlock S;
    I.o_T1 = S.take(16ull * r1);
    I.o_TQ1 = S.take(4ull * ES_FMAX * r1);
    I.o_D2 = S.take(16ull * r2);
    I.o_DQ2 = S.take(4ull * ES_FMAX * r2);
    I.o_S0 = S.take(16ull * (r0 + 1));   // + sentinel S0[r0] = M
    I.o_K0 = S.take(4ull * (r0 + 1));    // + sentinel K0[r0] = 0xffffffff
    I.o_I0 = S.take(4ull * r0);
    I.o_Q0 = S.take(4ull * ES_FMAX * r0);
    I.o_BK = S.take(16ull * (ES_NBUCKET + 1));
    I.o_FC = S.take(sizeof(EsFilterC) * std::max<uint32_t>(nf, 1));
    I.o_K1 = S.take(4ull * r1);
    for (uint32_t i = 0; i < r1; ++i) {
        const u128 v = P.terms[P.roff[1] + i];
        S.put128(I.o_T1, i, v);
        S.put32(I.o_K1, i, (uint32_t)(v >> sh));
        for (uint32_t f = 0; f < FB; ++f) S.put32(I.o_TQ1, i * ES_FMAX + f, es_mod(v, P.q[f]));
    }
    for (uint32_t i = 0; i < r2; ++i) {
        const u128 dlt = es_ring2_delta(P, i);
        S.put128(I.o_D2, i, dlt);
        for (uint32_t f = 0; f < FB; ++f) S.put32(I.o_DQ2, i * ES_FMAX + f, es_mod(dlt, P.q[f]));
    }
    for (uint32_t i = 0; i < r0; ++i) {
        S.put128(I.o_S0, i, R.S0[i]);
        S.put32(I.o_K0, i, K0[i]);
        S.put32(I.o_I0, i, R.digit[i]);
        for (uint32_t f = 0; f < FB; ++f) S.put32(I.o_Q0, (size_t)f * r0 + i, es_mod(R.S0[i], P.q[f]));
    }
    S.put128(I.o_S0, r0, M);             // stops the tie scan: M < thr never holds (thr <= M)
    S.put32(I.o_K0, r0, 0xffffffffu);    // stops the key scan: never < t32
    memcpy(&S.b[I.o_BK], BK.data(), 16ull * (ES_NBUCKET + 1));
    if (nf) memcpy(&S.b[I.o_FC], fc.data(), sizeof(EsFilterC) * nf);

    // ---- word-mask phase tables for the first FB filters ---------------------------------
    const uint32_t RS = es_row_words(W);
    std::vector<uint32_t> mask_off(ES_FMAX + 1, 0);
    for (uint32_t f = 0; f < ES_FMAX; ++f)
        mask_off[f + 1] = mask_off[f] + (f < FB ? (uint32_t)es_align_up((uint64_t)P.q[f] * RS, 4) : 0u);
    std::vector<uint32_t> masks(std::max<uint32_t>(mask_off[ES_FMAX], 4), 0u);
    std::vector<uint8_t> adm;
    for (uint32_t f = 0; f < FB; ++f) {
        const uint32_t q = P.q[f];
        adm.assign(q, 0);
        for (uint32_t r = 0; r < q; ++r) adm[r] = (P.allowed[P.bit_off[f] + (r >> 5)] >> (r & 31u)) & 1u;
        uint32_t* D = masks.data() + mask_off[f];
        for (uint32_t i = 0; i < r0; ++i) {
            const uint32_t a = es_mod(R.S0[i], q), wd = i >> 5, at = i & 31u;
            for (uint32_t ph = 0; ph < q - a; ++ph) D[(uint64_t)ph * RS + wd] |= (uint32_t)adm[ph + a] << at;
            for (uint32_t ph = q - a; ph < q; ++ph) D[(uint64_t)ph * RS + wd] |= (uint32_t)adm[ph + a - q] << at;
        }
    }
    // pair tables (inner rings of at most two words): phase row phi holds P_f[phi] and then the
    // row a wrap past M selects, P_f[(phi + corr_f) mod q_f], so one load serves both sides of
    // the carry split; filter f starts at word 2 * mask_off[f]
    std::vector<uint32_t> pairs;
    if (W <= 2) {
        pairs.assign(2ull * masks.size(), 0u);
        for (uint32_t f = 0; f < FB; ++f) {
            const uint32_t q = P.q[f], corr = fc[f].corr;
            const uint32_t* D0 = masks.data() + mask_off[f];
            uint32_t* D = pairs.data() + 2ull * mask_off[f];
            for (uint32_t ph = 0; ph < q; ++ph) {
                const uint32_t ph1 = ph + corr >= q ? ph + corr - q : ph + corr;
                for (uint32_t wd = 0; wd < W; ++wd) {
                    D[(uint64_t)ph * 2 * W + wd] = D0[(uint64_t)ph * W + wd];
                    D[(uint64_t)ph * 2 * W + W + wd] = D0[(uint64_t)ph1 * W + wd];
                }
            }
        }
    }
    I.F_built = FB;
    I.bsh = bsh;
    I.small_bytes = (uint32_t)S.b.size();
    for (uint32_t f = 0; f <= ES_FMAX; ++f) I.mask_off[f] = mask_off[f];
    I.mask_stride = RS;
    if (int e = upload_set(c, T, S.b, masks, pairs, P.allowed, P.terms)) return e;
    c->caller = T;
    return ES_OK;
}

// The host image of the production cascade with F inner tables.
static void prod_image(const es_ctx* c, uint32_t F, EsProdImage& img, double max_rate = 1.0) {
    // beside the staged tables: the static shared memory, and the slots of the largest CTA's warps
    es_prod_image(c->plan, c->geo, F,
                  (uint32_t)g_dev.smem_optin - 2048u - ES_PROD_THREADS / 32u * ES_QUEUE_BYTES, img, max_rate);
}

// Whether a CTA of any size has room for it (runs_production asks for the launch's own).
static bool image_fits(const EsProdImage& img) {
    return img.small.size() + es_align_up(4 * img.tabs.size(), 16) + ES_PROD_THREADS / 32u * ES_QUEUE_BYTES <=
           (size_t)g_dev.smem_optin - 1024u;
}

static int upload_prod(es_ctx* c, uint32_t F, EsProdImage& img) {
    TableSet T;
    T.h = img.inst;
    if (int e = upload_set(c, T, img.small, img.tabs, {}, img.bits, img.sums)) return e;
    c->prod[F].t = T;
    c->prod[F].entries = std::move(img.entries);
    return ES_OK;
}

// Candidates per warp-wide ring-1 digit above which a plan's own launches take one more inner table
// than asked for: the queue's passes then cost more than the table, which few lanes read.  A wider ring
// reads more of it, two rows of its words instead of one, so the line lies higher there.  With four
// tables and with five, 2^32 positions, us by candidates with four:
//   one word       0.28: 340, 354   0.44: 468, 460   0.51: 469, 436   0.80: 448, 429   1.09: 400, 368
//   two words      0.57: 516, 537   1.01: 373, 385   1.10: 391, 390   1.19: 387, 371   1.90: 481, 391
//   three or four  1.47: 358, 380   2.24: 360, 363   2.88: 432, 439   3.41: 393, 382   5.66: 430, 391
//   five and more  1.1 a word: 548, 595   1.6: 556, 621   2.1: 575, 644   2.5: 483, 428   4.4: 1228, 1003
// (k = 160..400 and the recorded wheels; for five and more words wheels of k = 220..390 around one large
// prime, of which 2.5 and 5.1 candidates a word also lost 4 and 10 %).
static double more_tables(uint32_t words) { return words == 1 ? 0.5 : words == 2 ? 1.15 : words <= 4 ? 3.2 : 2.3 * words; }

// Builds the table sets that launches of this shape read, unless they are there already: the
// plan's own launches (own), or those of a batch of several plans, which share a table count.
static int ensure_tables(es_ctx* c, const es_tune& t, bool own) {
    uint32_t F = prod_tables(t);
    if (own && !c->own_tables[F]) {
        EsProdImage img;
        uint32_t use = F;
        const double most = F < ES_PMAX ? more_tables(c->geo.W) / (32.0 * c->geo.r0) : 1.0;
        prod_image(c, F, img, most);
        if (img.rate > most) {
            prod_image(c, use = F + 1, img);
            if (!image_fits(img)) prod_image(c, use = F, img);   // (its ring-1 and step rows may be twice as long)
        }
        if (!c->prod[use].t.d)   // (counting contexts too: es_search_blocks_static never counts)
            if (int e = upload_prod(c, use, img)) return e;
        c->own_tables[F] = use;
    }
    if (own) F = c->own_tables[F];
    if (!c->prod[F].t.d) {
        EsProdImage img;
        prod_image(c, F, img);
        if (int e = upload_prod(c, F, img)) return e;
    }
    es_tune s = t;
    s.count_stages = 0;
    if ((!is_production(t) || !runs_production(c, s, F)) && !c->caller.d)
        if (int e = build_caller(c)) return e;
    return ES_OK;
}

int es_ctx_create(const es_plan_desc* d, const es_tune* tune_in, es_ctx** out) try {
    if (!d || !out) return fail(ES_ERR_ARG, "null descriptor or output pointer");
    *out = nullptr;
    es_tune tune = tune_in ? *tune_in : default_tune();
    if (int e = check_tune(tune)) return e;
    std::string bad;
    if (int code = es_check_desc(*d, bad)) return fail(code, bad);
    if (int e = device_facts()) return e;

    std::unique_ptr<es_ctx, int (*)(es_ctx*)> own(new es_ctx(), es_ctx_destroy);
    es_ctx* c = own.get();
    c->pool = BatchPool::of_device(g_dev.dev);
    std::string why;
    if (int code = es_parse_plan(*d, c->plan, c->geo, why)) return fail(code, why);
    const uint32_t nf = d->n_filters;
    c->tune = tune;
    c->M = c->plan.M;
    c->q = c->plan.q;
    if (int e = ensure_tables(c, tune, true)) return e;
    cudaError_t ce = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    if (ce == cudaSuccess) ce = cudaEventCreate(&c->ev0);
    if (ce == cudaSuccess) ce = cudaEventCreate(&c->ev1);
    if (ce == cudaSuccess) ce = cudaMalloc(&c->d_counts, 8ull * std::max<uint32_t>(nf, 1));
    if (ce == cudaSuccess) ce = cudaMalloc(&c->d_surv_n, 8ull * 8);
    if (ce == cudaSuccess) ce = cudaHostAlloc(&c->h_pin, 8ull * 8, cudaHostAllocDefault);
    // on the launches' own stream: nothing orders it after the default stream
    if (ce == cudaSuccess) ce = cudaMemsetAsync(c->d_counts, 0, 8ull * std::max<uint32_t>(nf, 1), c->stream);
    if (ce == cudaSuccess) ce = cudaMemsetAsync(c->d_surv_n, 0, 8ull * 8, c->stream);
    if (ce != cudaSuccess) return cuda_fail(ce, "context setup");
    // d_surv_n block: [0] survivor count, [1] unit counter, [2] CTAs done, [3..6] group min
    c->d_unit = c->d_surv_n + 1;
    c->d_done = c->d_surv_n + 2;
    c->d_min = c->d_surv_n + 3;
    if (int e = es_set_capacity(c, 1u << 20)) return e;
    *out = own.release();
    return ES_OK;
}
ES_CATCH

int es_cascade_image(const es_plan_desc* d, uint32_t tables, uint32_t smem_bytes, es_cascade_info* info, void* small,
                     uint64_t small_cap, uint32_t* tabs, uint64_t tabs_cap, uint32_t* parts, uint64_t parts_cap) try {
    if (!d || !info) return fail(ES_ERR_ARG, "null argument");
    if (tables < 1 || tables > ES_PMAX) return fail(ES_ERR_ARG, "tables must be in 1..6");
    std::string why;
    EsHostPlan P;
    EsInst geo{};
    if (int code = es_check_desc(*d, why)) return fail(code, why);
    if (int code = es_parse_plan(*d, P, geo, why)) return fail(code, why);
    EsProdImage img;
    es_prod_image(P, geo, tables, smem_bytes, img);
    const EsInst& I = img.inst;
    memset(info, 0, sizeof(*info));
    info->n_entries = I.n_filters;
    info->row_bytes = I.row_bytes;
    info->key_shift = I.sh;
    info->key_up = I.lsh;
    info->bucket_log2 = ES_PBUCKET_LOG2;
    info->o_row1 = I.o_R1;
    info->row1_bytes = tables <= 3 ? 16u : 32u;
    info->o_terms1 = I.o_T1;
    info->o_sorted = I.o_S0;
    info->o_digits = I.o_I0;
    info->o_buckets = I.o_BK;
    info->small_bytes = img.small.size();
    info->tab_words = img.tabs.size();
    for (uint32_t i = 0; i < tables; ++i) {
        info->tab_base[i] = I.tab_base[i];
        info->tab_wrap[i] = I.tab_wrap[i];
        info->tab_mul[i] = I.tab_mul[i];
    }
    uint64_t np = 0;
    for (uint32_t i = 0; i < img.entries.size(); ++i)
        for (const EsCascadeEntry::Part& p : img.entries[i].parts) {
            if (parts && 3 * np + 2 < parts_cap) {
                parts[3 * np] = i;
                parts[3 * np + 1] = p.f;
                parts[3 * np + 2] = p.d;
            }
            ++np;
        }
    info->n_parts = np;
    if (small && small_cap >= img.small.size()) memcpy(small, img.small.data(), img.small.size());
    if (tabs && tabs_cap >= img.tabs.size()) memcpy(tabs, img.tabs.data(), 4ull * img.tabs.size());
    return ES_OK;
}
ES_CATCH

int es_ctx_set_tune(es_ctx* c, const es_tune* t) try {
    if (!c || !t) return fail(ES_ERR_ARG, "null argument");
    if (int e = check_tune(*t)) return e;
    if (int e = ensure_tables(c, *t, true)) return e;
    c->tune = *t;
    return ES_OK;
}
ES_CATCH

int es_ctx_get_tune(const es_ctx* c, es_tune* t) {
    if (!c || !t) return fail(ES_ERR_ARG, "null argument");
    *t = c->tune;
    return ES_OK;
}

int es_ctx_info(const es_ctx* c, uint64_t* n_outer, uint32_t* r0, uint32_t* n_filters,
                uint64_t* table_bytes) {
    if (!c) return fail(ES_ERR_ARG, "null context");
    if (n_outer) *n_outer = c->geo.n_outer;
    if (r0) *r0 = c->geo.r0;
    if (n_filters) *n_filters = c->geo.n_filters;
    if (table_bytes) {
        *table_bytes = c->caller.bytes;
        for (const ProdSet& p : c->prod) *table_bytes += p.t.bytes;
    }
    return ES_OK;
}

int es_set_capacity(es_ctx* c, uint64_t cap) {
    if (!c || cap == 0 || cap > (1ull << 32)) return fail(ES_ERR_ARG, "capacity must be in [1, 2^32]");
    ES_CUDA(cudaStreamSynchronize(c->stream), "sync");
    cudaFree(c->d_surv);
    c->d_surv = nullptr;
    c->surv_cap = 0;   // until there is a new one, launches count and store nothing
    ES_CUDA(cudaMalloc(&c->d_surv, sizeof(es_survivor) * cap), "cudaMalloc(survivors)");
    c->surv_cap = cap;
    return ES_OK;
}

int es_set_block(es_ctx* c, const uint32_t* tconst, uint32_t n, uint64_t t) {
    if (!c) return fail(ES_ERR_ARG, "null context");
    if (n != c->geo.n_filters || (n && !tconst))
        return fail(ES_ERR_ARG, "tconst length must equal the number of filters");
    for (uint32_t f = 0; f < n; ++f) {
        if (tconst[f] >= c->q[f]) return fail(ES_ERR_ARG, "tconst[j] must be < q_j");
        c->tconst[f] = tconst[f];
    }
    c->t = t;
    return ES_OK;
}

int es_reset_survivors(es_ctx* c) {
    if (!c) return fail(ES_ERR_ARG, "null context");
    c->count_known = false;
    ES_CUDA(cudaMemsetAsync(c->d_surv_n, 0, 8, c->stream), "memset");
    return ES_OK;
}

int es_reset_counts(es_ctx* c) {
    if (!c) return fail(ES_ERR_ARG, "null context");
    ES_CUDA(cudaMemsetAsync(c->d_counts, 0, 8ull * std::max<uint32_t>(c->geo.n_filters, 1),
                            c->stream), "memset");
    return ES_OK;
}

static int ctx_launch(es_ctx* c, uint64_t ob, uint64_t oe, const uint64_t* d_list) {
    es_tune tn = c->tune;
    const uint32_t PF = c->own_tables[prod_tables(tn)];
    const bool prod = runs_production(c, tn, PF);
    if (prod) tn = prod_shape(tn);
    if (!prod && !tn.count_stages) tn.layout = ES_LAYOUT_SCALAR;
    const TableSet& T = prod ? c->prod[PF].t : c->caller;
    const EsInst& I = T.h;
    EsLaunch L;
    memset(&L, 0, sizeof(L));
    EsItem& it = L.item0;
    it.inst = T.d;
    it.tconst = nullptr;
    it.list = d_list;
    it.counts = tn.count_stages ? c->d_counts : nullptr;
    it.t = c->t;
    it.o_begin = ob;
    it.o_end = oe;
    uint64_t n_work;
    if (d_list) {
        it.c_begin = it.c_end = 0;
        n_work = oe - ob;
    } else {
        n_work = cycles_of(I, ob, oe, &it.c_begin);
        it.c_end = it.c_begin + n_work;
    }
    tn.strip = launch_strip(
        d_list ? (n_work + 31) / 32 : steps_of(I, it.c_begin, it.c_end), tn,
        [&](uint32_t w) {
            return d_list ? (n_work + 32ull * w - 1) / (32ull * w) : units_of(I, it.c_begin, it.c_end, w);
        },
        [&](uint32_t w) { return d_list ? w : longest_of(I, w); });
    const uint64_t per_unit = 32ull * tn.strip;
    it.unit_begin = 0;
    it.n_units = d_list ? (n_work + per_unit - 1) / per_unit : units_of(I, it.c_begin, it.c_end, tn.strip);
    it.group = 0;
    it.inst_id = 0;
    const uint32_t F = prod ? PF : stage_filters(tn.layout, tn.mask_filters, I.n_filters, I.F_built);
    const uint32_t layout = prod ? ES_LAYOUT_PROD
                                 : launch_layout(tn.layout, I.W, I.small_bytes, I.n_filters, tn, I.mask_off[F]);
    const SmemPlan sp = plan_smem((uint32_t)I.small_bytes, I.n_filters, tn,
                                  prod ? I.tab_words : staged_words(layout, I.mask_off[F]));
    it.caller = 0;
    L.items = nullptr;
    L.n_items = 1;
    L.threads = tn.threads;
    L.strip = tn.strip;
    L.mask_filters = F;
    L.total_units = it.n_units;
    L.nf_max = std::max<uint32_t>(I.n_filters, 1);
    L.direct = 1;
    L.unit_counter = c->d_unit;
    L.ctas_done = c->d_done;
    L.surv = c->d_surv;
    L.surv_n = c->d_surv_n;
    L.surv_cap = c->surv_cap;
    L.group_found = nullptr;
    L.smem_bytes = sp.bytes;
    L.cnt_off = sp.cnt_off;
    L.queue_off = sp.queue_off;
    L.stage_off = sp.stage_off;
    launch_tables(L, I);
    if (prod)
        prod_tconst(c->prod[PF], c->tconst, L.tconst0);
    else
        memcpy(L.tconst0, c->tconst, 4ull * I.n_filters);
    if (it.n_units == 0) return ES_OK;
    int grid = 0;
    if (int e = grid_for(layout, tn.count_stages, I.W, F, tn, sp.bytes, it.n_units, &grid)) return e;
    c->count_known = false;
    int e = es_launch_scan(L, (int)layout, (int)tn.count_stages, I.W, grid, c->stream);
    if (e) return cuda_fail((cudaError_t)e, "scan launch");
    return ES_OK;
}

int es_launch(es_ctx* c, uint64_t ostart, uint64_t ocount) {
    if (!c) return fail(ES_ERR_ARG, "null context");
    if (ostart > c->geo.n_outer || ocount > c->geo.n_outer - ostart)
        return fail(ES_ERR_RANGE, "outer range outside [0, R/r0)");
    return ctx_launch(c, ostart, ostart + ocount, nullptr);
}

int es_launch_list(es_ctx* c, const uint64_t* outer, uint64_t n) {
    if (!c || (n && !outer)) return fail(ES_ERR_ARG, "null argument");
    for (uint64_t i = 0; i < n; ++i)
        if (outer[i] >= c->geo.n_outer) return fail(ES_ERR_RANGE, "outer index outside [0, R/r0)");
    if (n == 0) return ES_OK;
    ES_CUDA(cudaStreamSynchronize(c->stream), "sync");
    if (n > c->list_cap) {
        cudaFree(c->d_list);
        c->d_list = nullptr;
        c->list_cap = 0;
        ES_CUDA(cudaMalloc(&c->d_list, 8ull * n), "cudaMalloc(list)");
        c->list_cap = n;
    }
    ES_CUDA(cudaMemcpyAsync(c->d_list, outer, 8ull * n, cudaMemcpyHostToDevice, c->stream), "copy list");
    ES_CUDA(cudaStreamSynchronize(c->stream), "copy list");   // the caller's array has been read
    return ctx_launch(c, 0, n, c->d_list);
}

int es_sync(es_ctx* c) {
    if (!c) return fail(ES_ERR_ARG, "null context");
    ES_CUDA(cudaStreamSynchronize(c->stream), "kernel execution");
    return ES_OK;
}

int es_survivor_count(es_ctx* c, uint64_t* n) {
    if (!c || !n) return fail(ES_ERR_ARG, "null argument");
    if (!c->count_known) {
        ES_CUDA(cudaMemcpyAsync(c->h_pin, c->d_surv_n, 8, cudaMemcpyDeviceToHost, c->stream), "copy");
        ES_CUDA(cudaStreamSynchronize(c->stream), "kernel execution");
        c->count = c->h_pin[0];
        c->count_known = true;
    }
    *n = c->count;
    return ES_OK;
}

int es_read_survivor_records(es_ctx* c, es_survivor* out, uint64_t cap, uint64_t* n) {
    if (!c || !n) return fail(ES_ERR_ARG, "null argument");
    uint64_t cnt = 0;
    if (int e = es_survivor_count(c, &cnt)) return e;
    *n = cnt;
    if (cnt > c->surv_cap)
        return fail(ES_ERR_OVERFLOW, "survivor buffer overflow (" + std::to_string(cnt) + " > " +
                                         std::to_string(c->surv_cap) + "); raise max_survivors");
    if (cnt > cap) return fail(ES_ERR_OVERFLOW, "output buffer smaller than the survivor count");
    if (cnt) ES_CUDA(cudaMemcpy(out, c->d_surv, sizeof(es_survivor) * cnt, cudaMemcpyDeviceToHost), "copy");
    return ES_OK;
}

int es_read_survivors(es_ctx* c, uint64_t* idx_out, uint64_t cap, uint64_t* n) try {
    if (!c || !n) return fail(ES_ERR_ARG, "null argument");
    uint64_t cnt = 0;
    if (int e = es_survivor_count(c, &cnt)) return e;
    *n = cnt;
    if (cnt > c->surv_cap)
        return fail(ES_ERR_OVERFLOW, "survivor buffer overflow (" + std::to_string(cnt) + " > " +
                                         std::to_string(c->surv_cap) + "); raise max_survivors");
    if (cnt > cap) return fail(ES_ERR_OVERFLOW, "output buffer smaller than the survivor count");
    if (!cnt) return ES_OK;
    std::vector<es_survivor> tmp(cnt);
    ES_CUDA(cudaMemcpy(tmp.data(), c->d_surv, sizeof(es_survivor) * cnt, cudaMemcpyDeviceToHost), "copy");
    for (uint64_t i = 0; i < cnt; ++i) idx_out[i] = tmp[i].idx;
    return ES_OK;
}
ES_CATCH

int es_stage_counts(es_ctx* c, uint64_t* counts, uint32_t n) {
    if (!c || (n && !counts)) return fail(ES_ERR_ARG, "null argument");
    if (n != c->geo.n_filters) return fail(ES_ERR_ARG, "counts length must equal the filter count");
    ES_CUDA(cudaStreamSynchronize(c->stream), "kernel execution");
    if (n) ES_CUDA(cudaMemcpy(counts, c->d_counts, 8ull * n, cudaMemcpyDeviceToHost), "copy");
    return ES_OK;
}

int es_min_survivor(es_ctx* c, int* found, uint64_t* t, uint64_t* s_lo, uint64_t* s_hi) {
    if (!c || !found) return fail(ES_ERR_ARG, "null argument");
    int e = es_launch_min(c->d_surv, c->d_surv_n, c->surv_cap, nullptr, 1, nullptr, c->d_min, c->stream);
    if (e) return cuda_fail((cudaError_t)e, "min launch");
    ES_CUDA(cudaMemcpyAsync(c->h_pin, c->d_min, 32, cudaMemcpyDeviceToHost, c->stream), "copy");
    ES_CUDA(cudaStreamSynchronize(c->stream), "kernel execution");
    if (c->h_pin[0] == 2)
        return fail(ES_ERR_OVERFLOW, "survivor buffer overflow: the minimum over the stored records "
                                     "is not reliable; raise the capacity or scan fewer positions");
    *found = (int)c->h_pin[0];
    if (t) *t = c->h_pin[1];
    if (s_lo) *s_lo = c->h_pin[2];
    if (s_hi) *s_hi = c->h_pin[3];
    return ES_OK;
}

int es_launch_timed(es_ctx* c, uint64_t ostart, uint64_t ocount, float* ms) {
    if (!c) return fail(ES_ERR_ARG, "null context");
    ES_CUDA(cudaEventRecord(c->ev0, c->stream), "event");
    if (int e = es_launch(c, ostart, ocount)) return e;
    ES_CUDA(cudaEventRecord(c->ev1, c->stream), "event");
    ES_CUDA(cudaEventSynchronize(c->ev1), "kernel execution");
    float v = 0.f;
    ES_CUDA(cudaEventElapsedTime(&v, c->ev0, c->ev1), "event");
    if (ms) *ms = v;
    return ES_OK;
}

// ---------------------------------------------------------------------------------------
int es_batch_destroy(es_batch* b) {
    if (!b) return ES_OK;
    if (b->stream) cudaStreamSynchronize(b->stream);
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    if (b->mem && b->pool) b->pool->give(std::move(b->mem));
    delete b;
    return ES_OK;
}

int es_batch_create(es_ctx* const* ctxs, uint32_t n_ctx, const es_batch_item* items,
                    uint32_t n_items, const es_tune* tune_in, es_batch** out) try {
    if (!ctxs || !items || !out || n_ctx == 0 || n_items == 0)
        return fail(ES_ERR_ARG, "empty batch");
    *out = nullptr;
    es_tune tune = tune_in ? *tune_in : ctxs[0]->tune;
    if (int e = check_tune(tune)) return e;
    if (int e = device_facts()) return e;
    std::unique_ptr<es_batch, int (*)(es_batch*)> own(new es_batch(), es_batch_destroy);
    es_batch* b = own.get();
    b->tune = tune;
    b->ctxs.assign(ctxs, ctxs + n_ctx);
    for (uint32_t i = 0; i < n_ctx; ++i) {
        if (!ctxs[i]) return fail(ES_ERR_ARG, "null context in batch");
        if (int e = ensure_tables(ctxs[i], tune, n_ctx == 1)) return e;
    }
    const uint32_t PF = n_ctx == 1 ? ctxs[0]->own_tables[prod_tables(tune)] : prod_tables(tune);
    // the table set a plan's items run on
    auto tables = [&](const es_ctx* c) -> const TableSet& {
        return runs_production(c, tune, PF) ? c->prod[PF].t : c->caller;
    };
    // width class of a plan: the kernel instance its inner ring uses
    auto width_class = [](uint32_t W) -> uint32_t { return W <= 2 ? W : (W <= 4 ? 4u : 0u); };
    std::vector<uint32_t> h_tc;
    b->h_items.resize(n_items);
    b->count_off.resize(n_items);
    uint64_t cwords = 0;
    uint32_t max_group = 0;
    for (uint32_t i = 0; i < n_items; ++i) {
        const es_batch_item& s = items[i];
        if (s.ctx_index >= n_ctx) return fail(ES_ERR_ARG, "item ctx_index out of range");
        if (s.group >= n_items) return fail(ES_ERR_ARG, "item group must be < n_items");
        const es_ctx* c = ctxs[s.ctx_index];
        const EsInst& I = c->geo;
        if (s.o_begin > s.o_end || s.o_end > I.n_outer)
            return fail(ES_ERR_RANGE, "item outer range outside [0, R/r0)");
        EsItem& it = b->h_items[i];
        memset(&it, 0, sizeof(it));
        it.inst = tables(c).d;
        it.list = nullptr;
        it.t = s.t;
        it.o_begin = s.o_begin;
        it.o_end = s.o_end;
        const uint64_t ncyc = s.o_end > s.o_begin ? cycles_of(I, s.o_begin, s.o_end, &it.c_begin) : 0;
        it.c_end = it.c_begin + ncyc;
        it.group = s.group;
        it.inst_id = s.ctx_index;
        it.caller = i;
        // per-block constants, in the order of the table set's entries
        it.tconst = reinterpret_cast<const uint32_t*>((uintptr_t)h_tc.size());  // patched below
        uint32_t caller_tc[ES_MAX_FILTERS], entry_tc[ES_MAX_ENTRIES];
        block_tconst(c, s.t, caller_tc);
        const bool prod = runs_production(c, tune, PF);
        if (prod) prod_tconst(c->prod[PF], caller_tc, entry_tc);
        h_tc.insert(h_tc.end(), prod ? entry_tc : caller_tc,
                    prod ? entry_tc + c->prod[PF].entries.size() : caller_tc + I.n_filters);
        while (h_tc.size() % 4) h_tc.push_back(0);
        b->count_off[i] = cwords;
        cwords += std::max<uint32_t>(I.n_filters, 1);
        max_group = std::max<uint32_t>(max_group, s.group);
    }
    b->n_groups = max_group + 1;
    // launch order: items grouped by width class (stable), one launch per class; counting launches
    // with ES_LAYOUT_AUTO split a one- or two-word class further into the plans whose inner-stage
    // tables fit shared memory (staged) and the rest
    auto class_key = [&](uint32_t item) -> uint32_t {
        const EsInst& I = tables(ctxs[items[item].ctx_index]).h;
        uint32_t key = 2u * width_class(I.W);
        if (!tune.count_stages) return key + (runs_production(ctxs[items[item].ctx_index], tune, PF) ? 1u : 0u);
        if (tune.layout == ES_LAYOUT_AUTO && (I.W == 1 || I.W == 2)) {
            const uint32_t Fi = stage_filters(tune.layout, tune.mask_filters, I.n_filters, I.F_built);
            if (launch_layout(ES_LAYOUT_AUTO, I.W, (uint32_t)I.small_bytes, I.n_filters, tune, I.mask_off[Fi]) ==
                ES_LAYOUT_SMEM)
                key += 1u;
        }
        return key;
    };
    std::vector<uint32_t> keys(n_items);
    for (uint32_t i = 0; i < n_items; ++i) keys[i] = class_key(i);
    std::vector<uint32_t> order(n_items);
    for (uint32_t i = 0; i < n_items; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return keys[x] < keys[y]; });
    // device block: items (caller order, launch order), constants (uploaded in one copy), scalars
    const size_t items_bytes = es_align_up(sizeof(EsItem) * n_items, 16);
    const size_t upload = 2 * items_bytes + es_align_up(4ull * h_tc.size(), 16);
    const size_t n_scalars = 4ull * b->n_groups + 1 + 2ull * n_items + cwords + b->n_groups;
    b->pool = ctxs[0]->pool;
    b->mem = b->pool->take(ctxs[0]->surv_cap);
    if (!b->mem) b->mem.reset(new BatchMem());
    b->surv_cap = ctxs[0]->surv_cap;
    cudaError_t ce = b->mem->need(upload + 8 * n_scalars, upload + 8 * (4ull * b->n_groups + 1), b->surv_cap);
    if (ce != cudaSuccess) {
        b->mem.reset();
        return cuda_fail(ce, "batch setup");
    }
    b->stream = b->mem->stream;
    b->ev0 = b->mem->ev0;
    b->ev1 = b->mem->ev1;
    b->d_surv = b->mem->surv;
    b->d_items = reinterpret_cast<EsItem*>(b->mem->dev);
    b->d_items_launch = reinterpret_cast<EsItem*>(b->mem->dev + items_bytes);
    b->d_tconst = reinterpret_cast<uint32_t*>(b->mem->dev + 2 * items_bytes);
    b->d_min = reinterpret_cast<unsigned long long*>(b->mem->dev + upload);
    b->d_surv_n = b->d_min + 4ull * b->n_groups;
    b->d_unit = b->d_surv_n + 1;
    b->d_item_next = b->d_unit + n_items;
    b->d_counts = b->d_item_next + n_items;
    b->d_found = b->d_counts + cwords;
    b->zero_bytes = 8ull * (size_t)(b->d_found - b->d_surv_n);
    b->h_result = reinterpret_cast<unsigned long long*>(b->mem->pin + upload);
    b->n_items = n_items;
    for (uint32_t i = 0; i < n_items; ++i) {
        EsItem& it = b->h_items[i];
        it.tconst = b->d_tconst + (uintptr_t)it.tconst;
        it.counts = tune.count_stages ? b->d_counts + b->count_off[i] : nullptr;
    }
    // the launches, one per width class, each over its own unit space
    std::vector<EsItem> launch_items(n_items);
    uint32_t pos = 0;
    while (pos < n_items) {
        const uint32_t first_ctx = items[order[pos]].ctx_index;
        const uint32_t cls = width_class(ctxs[first_ctx]->geo.W);
        uint32_t end = pos, small_max = 0, nf_max = 1, stage_max = 0;
        const bool prod = runs_production(ctxs[first_ctx], tune, PF);
        const uint32_t layout = prod || tune.count_stages ? tune.layout : (uint32_t)ES_LAYOUT_SCALAR;
        uint32_t F = prod ? PF : tune.mask_filters;
        bool one_ctx = true;
        uint32_t words = ctxs[first_ctx]->geo.W;
        uint64_t units = 0, steps = 0;
        es_tune shape = prod ? prod_shape(tune) : tune;
        while (end < n_items && keys[order[end]] == keys[order[pos]]) {
            const uint32_t ci = items[order[end]].ctx_index;
            const EsInst& I = tables(ctxs[ci]).h;
            const uint32_t small = std::max<uint32_t>(small_max, I.small_bytes);
            if (prod) {
                // plans that fit a CTA's shared memory one by one may not fit it together
                const uint32_t stage = std::max(stage_max, I.tab_words);
                if (end > pos && plan_smem(small, 1, shape, stage).bytes > (uint32_t)g_dev.smem_optin - 1024u) break;
                stage_max = stage;
            } else {
                F = std::min(F, stage_filters(layout, tune.mask_filters, I.n_filters, I.F_built));
            }
            small_max = small;
            nf_max = std::max<uint32_t>(nf_max, I.n_filters);
            if (ci != first_ctx) one_ctx = false;
            if (I.W != words) words = 0;   // the generic instance reads each plan's width
            const EsItem& it = b->h_items[order[end]];
            steps += steps_of(I, it.c_begin, it.c_end);
            ++end;
        }
        auto geo_of = [&](uint32_t j) -> const EsInst& { return ctxs[items[order[j]].ctx_index]->geo; };
        shape.strip = launch_strip(
            steps, shape,
            [&](uint32_t w) {
                uint64_t n = 0;
                for (uint32_t j = pos; j < end; ++j)
                    n += units_of(geo_of(j), b->h_items[order[j]].c_begin, b->h_items[order[j]].c_end, w);
                return n;
            },
            [&](uint32_t w) {
                uint32_t m = 0;
                for (uint32_t j = pos; j < end; ++j) m = std::max(m, longest_of(geo_of(j), w));
                return m;
            });
        for (uint32_t j = pos; j < end; ++j) {
            EsItem& it = launch_items[j];
            it = b->h_items[order[j]];
            it.n_units = units_of(ctxs[items[order[j]].ctx_index]->geo, it.c_begin, it.c_end, shape.strip);
            it.unit_begin = units;
            units += it.n_units;
        }
        es_batch::Sub sub;
        sub.words = cls == 0 ? 0u : (cls == 4 && words == 0 ? 4u : (words ? words : cls));
        if (prod) {
            sub.layout = ES_LAYOUT_PROD;
        } else {
            uint32_t mask_words = 0;   // the largest inner-stage word-mask tables among the class's plans
            for (uint32_t j = pos; j < end; ++j)
                mask_words = std::max<uint32_t>(mask_words, tables(ctxs[items[order[j]].ctx_index]).h.mask_off[F]);
            sub.layout = launch_layout(layout, sub.words, small_max, nf_max, shape, mask_words);
            stage_max = staged_words(sub.layout, mask_words);
        }
        const SmemPlan sp = plan_smem(small_max, nf_max, shape, stage_max);
        EsLaunch& L = sub.L;
        memset(&L, 0, sizeof(L));
        L.items = b->d_items_launch + pos;
        L.n_items = end - pos;
        L.threads = shape.threads;
        L.strip = shape.strip;
        L.mask_filters = F;
        L.total_units = units;
        L.nf_max = nf_max;
        L.direct = one_ctx ? 1u : 0u;
        L.unit_counter = b->d_unit + b->subs.size();
        L.item_next = b->d_item_next + pos;
        L.surv = b->d_surv;
        L.surv_n = b->d_surv_n;
        L.surv_cap = b->surv_cap;
        L.group_found = b->d_found;
        L.smem_bytes = sp.bytes;
        L.cnt_off = sp.cnt_off;
        L.queue_off = sp.queue_off;
        L.stage_off = sp.stage_off;
        if (one_ctx) launch_tables(L, tables(ctxs[first_ctx]).h);
        if (int e = grid_for(sub.layout, tune.count_stages, sub.words, F, shape, sp.bytes,
                             std::max<uint64_t>(units, 1), &sub.grid))
            return e;
        b->subs.push_back(sub);
        pos = end;
    }
    unsigned char* stage = b->mem->pin;   // not written again before this batch's memory is reused
    memcpy(stage, b->h_items.data(), sizeof(EsItem) * n_items);
    memcpy(stage + items_bytes, launch_items.data(), sizeof(EsItem) * n_items);
    if (!h_tc.empty()) memcpy(stage + 2 * items_bytes, h_tc.data(), 4ull * h_tc.size());
    ce = cudaMemcpyAsync(b->mem->dev, stage, upload, cudaMemcpyHostToDevice, b->stream);
    if (ce != cudaSuccess) return cuda_fail(ce, "batch upload");
    *out = own.release();
    return ES_OK;
}
ES_CATCH

static int batch_enqueue(es_batch* b) {
    ES_CUDA(cudaMemsetAsync(b->d_surv_n, 0, b->zero_bytes, b->stream), "memset");
    ES_CUDA(cudaMemsetAsync(b->d_found, 0xff, 8ull * b->n_groups, b->stream), "memset");
    for (const es_batch::Sub& sub : b->subs) {
        if (!sub.L.total_units) continue;
        int e = es_launch_scan(sub.L, (int)sub.layout, (int)b->tune.count_stages, sub.words, sub.grid, b->stream);
        if (e) return cuda_fail((cudaError_t)e, "scan launch");
    }
    // survivors carry the caller's item index: the min-reduction reads the items in that order
    int e = es_launch_min(b->d_surv, b->d_surv_n, b->surv_cap, b->d_items, b->n_groups, b->d_found,
                          b->d_min, b->stream);
    if (e) return cuda_fail((cudaError_t)e, "min launch");
    ES_CUDA(cudaMemcpyAsync(b->h_result, b->d_min, 8ull * (4ull * b->n_groups + 1), cudaMemcpyDeviceToHost, b->stream),
            "copy");
    return ES_OK;
}

int es_batch_run(es_batch* b, int use_graph) {
    if (!b) return fail(ES_ERR_ARG, "null batch");
    ES_CUDA(cudaEventRecord(b->ev0, b->stream), "event");
    if (use_graph) {
        if (!b->exec) {
            ES_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal), "capture");
            int e = batch_enqueue(b);
            cudaGraph_t g = nullptr;
            cudaError_t ce = cudaStreamEndCapture(b->stream, &g);
            if (e) { if (g) cudaGraphDestroy(g); return e; }
            if (ce != cudaSuccess) return cuda_fail(ce, "end capture");
            b->graph = g;
            ES_CUDA(cudaGraphInstantiate(&b->exec, g, 0), "graph instantiate");
        }
        ES_CUDA(cudaGraphLaunch(b->exec, b->stream), "graph launch");
    } else {
        if (int e = batch_enqueue(b)) return e;
    }
    ES_CUDA(cudaEventRecord(b->ev1, b->stream), "event");
    b->ran = true;
    return ES_OK;
}

int es_batch_sync(es_batch* b, float* ms) {
    if (!b) return fail(ES_ERR_ARG, "null batch");
    ES_CUDA(cudaStreamSynchronize(b->stream), "kernel execution");
    if (ms) {
        float v = 0.f;
        if (b->ran) ES_CUDA(cudaEventElapsedTime(&v, b->ev0, b->ev1), "event");
        *ms = v;
    }
    return ES_OK;
}

int es_batch_group_min(es_batch* b, uint32_t group, int* found, uint64_t* t, uint64_t* s_lo,
                       uint64_t* s_hi) {
    if (!b || !found) return fail(ES_ERR_ARG, "null argument");
    if (group >= b->n_groups) return fail(ES_ERR_ARG, "group out of range");
    if (!b->ran) return fail(ES_ERR_STATE, "batch has not run");
    ES_CUDA(cudaStreamSynchronize(b->stream), "kernel execution");
    const unsigned long long* v = b->h_result + 4ull * group;
    *found = (int)v[0];
    if (t) *t = v[1];
    if (s_lo) *s_lo = v[2];
    if (s_hi) *s_hi = v[3];
    if (v[0] == 2)   // records were dropped: the minimum over the stored ones is not reliable
        return fail(ES_ERR_OVERFLOW, "survivor buffer overflow in the batch; the least block of this "
                                     "group holding a good survivor is t = " +
                                     (v[1] == ~0ull ? std::string("none") : std::to_string(v[1])) +
                                     "; rescan the group's blocks one at a time");
    return ES_OK;
}

int es_batch_item_counts(es_batch* b, uint32_t item, uint64_t* counts, uint32_t n) {
    if (!b || (n && !counts)) return fail(ES_ERR_ARG, "null argument");
    if (item >= b->h_items.size()) return fail(ES_ERR_ARG, "item out of range");
    const uint32_t nf = b->ctxs[b->h_items[item].inst_id]->geo.n_filters;
    if (n != nf) return fail(ES_ERR_ARG, "counts length must equal the item's filter count");
    if (!b->ran) return fail(ES_ERR_STATE, "batch has not run");
    ES_CUDA(cudaStreamSynchronize(b->stream), "kernel execution");
    if (n) ES_CUDA(cudaMemcpy(counts, b->d_counts + b->count_off[item], 8ull * n, cudaMemcpyDeviceToHost), "copy");
    return ES_OK;
}

int es_batch_survivors(es_batch* b, es_survivor* out, uint64_t cap, uint64_t* n) {
    if (!b || !n) return fail(ES_ERR_ARG, "null argument");
    if (!b->ran) return fail(ES_ERR_STATE, "batch has not run");
    ES_CUDA(cudaStreamSynchronize(b->stream), "kernel execution");
    const unsigned long long cnt = b->h_result[4ull * b->n_groups];
    *n = cnt;
    if (cnt > b->surv_cap) return fail(ES_ERR_OVERFLOW, "survivor buffer overflow");
    if (cnt > cap) return fail(ES_ERR_OVERFLOW, "output buffer smaller than the survivor count");
    if (cnt) ES_CUDA(cudaMemcpy(out, b->d_surv, sizeof(es_survivor) * cnt, cudaMemcpyDeviceToHost), "copy");
    return ES_OK;
}

static int int_peak_probe(int mix, double* ops_per_s, double* ms_out) {
    if (int e = device_facts()) return e;
    unsigned long long* sink = nullptr;
    ES_CUDA(cudaMalloc(&sink, 8), "cudaMalloc");
    cudaEvent_t a, z;
    cudaEventCreate(&a);
    cudaEventCreate(&z);
    const int threads = 256, grid = g_dev.sms * 8, iters = 4096;
    float best = 1e30f;
    for (int rep = 0; rep < 4; ++rep) {
        cudaEventRecord(a);
        int e = es_launch_int_peak(sink, grid, threads, iters, mix, nullptr);
        cudaEventRecord(z);
        cudaError_t ce = cudaEventSynchronize(z);
        if (e || ce != cudaSuccess) {
            cudaFree(sink);
            cudaEventDestroy(a);
            cudaEventDestroy(z);
            return cuda_fail(e ? (cudaError_t)e : ce, "int peak kernel");
        }
        float v = 0.f;
        cudaEventElapsedTime(&v, a, z);
        if (rep > 0 && v < best) best = v;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(z);
    cudaFree(sink);
    const double ops = (double)grid * threads * (double)iters * 256.0;
    if (ops_per_s) *ops_per_s = ops / (best * 1e-3);
    if (ms_out) *ms_out = best;
    return ES_OK;
}

int es_int_peak(double* ops_per_s, double* ms_out) { return int_peak_probe(0, ops_per_s, ms_out); }

int es_int_peak_mixed(double* ops_per_s, double* ms_out) { return int_peak_probe(1, ops_per_s, ms_out); }

}  // extern "C"

// ------------------------------------------------------------------------------------------
// es_search_blocks_static: the one entry point that allocates nothing.
//
// Some callers cannot call cudaMalloc at all: code running under an external memory manager
// (a framework that owns every device allocation, a pool with a hard budget), or a service
// that must not allocate after start-up.  For them this is a variant of the block-ordered
// multi-block search launch: blocks t0 .. t0+n_blocks-1 of an existing context, scanned in
// one persistent launch, the first block holding a good survivor ending the search.  The
// caller passes the inputs (the context's plan tables, built earlier) and the outputs (a
// survivor buffer, its count and the 4-word minimum).  The launch's scratch -- work counter,
// search flag, per-block item descriptors and block constants -- lives in the file-scope
// array below, of fixed size ES_STATIC_MAX_BLOCKS blocks x ES_MAX_ENTRIES entries (about
// 60 KB); every GPU that loads this library keeps it until the process exits.
namespace {

constexpr size_t kStaticItemsOff = 256;
constexpr size_t kStaticTconstOff = kStaticItemsOff + sizeof(EsItem) * ES_STATIC_MAX_BLOCKS;
constexpr size_t kStaticBytes = kStaticTconstOff + 4ull * ES_STATIC_MAX_BLOCKS * ES_MAX_ENTRIES;

// [0,8) work counter, [8,16) least block with a good survivor, items, per-block constants
static __device__ __align__(256) unsigned char g_static_scratch[kStaticBytes];

// Host side: the device address of g_static_scratch per device (the host symbol itself is
// only a stand-in and must never be passed to a kernel), and a host staging area for the
// descriptors (static storage: no heap allocation on the call path).
constexpr int kMaxDevices = 64;
unsigned char* g_static_ptr[kMaxDevices] = {nullptr};
EsItem g_static_items[ES_STATIC_MAX_BLOCKS];
uint32_t g_static_tconst[ES_STATIC_MAX_BLOCKS * ES_MAX_ENTRIES];
std::mutex g_static_mu;

}  // namespace

extern "C" int es_search_blocks_static(const es_ctx* c, uint64_t t0, uint32_t n_blocks,
                                       es_survivor* d_out, uint64_t out_cap,
                                       unsigned long long* d_count, unsigned long long* d_min,
                                       void* stream) {
    if (!c || !d_out || !d_count || !d_min || out_cap == 0)
        return fail(ES_ERR_ARG, "null context/output or zero output capacity");
    if (n_blocks == 0 || n_blocks > ES_STATIC_MAX_BLOCKS)
        return fail(ES_ERR_RANGE, "n_blocks must be in [1, " + std::to_string(ES_STATIC_MAX_BLOCKS) +
                                      "] for the static-scratch search");
    if (t0 > UINT64_MAX - n_blocks) return fail(ES_ERR_RANGE, "block range overflows");
    // the search never counts: the production cascade, or the scalar layout on request
    es_tune tn = c->tune;
    tn.count_stages = 0;
    const uint32_t PF = c->own_tables[prod_tables(tn)];
    const bool prod = runs_production(c, tn, PF);
    if (prod) tn = prod_shape(tn);
    const TableSet& T = prod ? c->prod[PF].t : c->caller;
    const EsInst& I = T.h;
    cudaStream_t st = (cudaStream_t)stream;
    // The descriptors below are copied from host staging arrays that the next call overwrites; a
    // captured copy would read them only when the graph runs, so capture is refused.
    cudaStreamCaptureStatus cap_status = cudaStreamCaptureStatusNone;
    ES_CUDA(cudaStreamIsCapturing(st, &cap_status), "cudaStreamIsCapturing");
    if (cap_status != cudaStreamCaptureStatusNone)
        return fail(ES_ERR_STATE, "es_search_blocks_static cannot be called while its stream is capturing");
    int dev = 0;
    ES_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev < 0 || dev >= kMaxDevices) return fail(ES_ERR_RANGE, "device index out of range");
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[dev]) {
        // once per device, with that device current: the scratch array's device address
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(static scratch)");
        g_static_ptr[dev] = static_cast<unsigned char*>(p);
    }
    unsigned char* base = g_static_ptr[dev];
    unsigned long long* d_unit = reinterpret_cast<unsigned long long*>(base);
    unsigned long long* d_found = d_unit + 1;
    EsItem* d_items = reinterpret_cast<EsItem*>(base + kStaticItemsOff);
    uint32_t* d_tc = reinterpret_cast<uint32_t*>(base + kStaticTconstOff);

    const uint32_t nf = I.n_filters;
    const uint32_t F = prod ? PF : stage_filters(tn.layout, tn.mask_filters, nf, I.F_built);
    const uint32_t layout = prod ? ES_LAYOUT_PROD : (uint32_t)ES_LAYOUT_SCALAR;
    const SmemPlan sp = plan_smem((uint32_t)I.small_bytes, nf, tn, prod ? I.tab_words : 0u);
    uint64_t cbeg = 0;
    const uint64_t ncyc = cycles_of(I, 0, I.n_outer, &cbeg);
    tn.strip = launch_strip(steps_of(I, cbeg, cbeg + ncyc) * n_blocks, tn,
                            [&](uint32_t w) { return units_of(I, cbeg, cbeg + ncyc, w) * n_blocks; },
                            [&](uint32_t w) { return longest_of(I, w); });
    const uint64_t nu = units_of(I, cbeg, cbeg + ncyc, tn.strip);
    for (uint32_t i = 0; i < n_blocks; ++i) {
        const uint64_t t = t0 + i;
        EsItem& it = g_static_items[i];
        memset(&it, 0, sizeof(it));
        it.inst = T.d;
        it.tconst = d_tc + (size_t)i * ES_MAX_ENTRIES;
        it.t = t;
        it.o_begin = 0;
        it.o_end = I.n_outer;
        it.c_begin = cbeg;
        it.c_end = cbeg + ncyc;
        it.unit_begin = nu * i;
        it.n_units = nu;
        it.caller = i;
        uint32_t* tc = g_static_tconst + (size_t)i * ES_MAX_ENTRIES;
        if (prod) {
            uint32_t caller_tc[ES_MAX_FILTERS];
            block_tconst(c, t, caller_tc);
            prod_tconst(c->prod[PF], caller_tc, tc);
        } else {
            block_tconst(c, t, tc);
        }
    }
    ES_CUDA(cudaMemcpyAsync(d_items, g_static_items, sizeof(EsItem) * n_blocks, cudaMemcpyHostToDevice, st),
            "copy items");
    ES_CUDA(cudaMemcpyAsync(d_tc, g_static_tconst, 4ull * ES_MAX_ENTRIES * n_blocks, cudaMemcpyHostToDevice, st),
            "copy block constants");
    ES_CUDA(cudaMemsetAsync(d_unit, 0, 8, st), "memset");
    ES_CUDA(cudaMemsetAsync(d_found, 0xff, 8, st), "memset");
    ES_CUDA(cudaMemsetAsync(d_count, 0, 8, st), "memset");

    EsLaunch L;
    memset(&L, 0, sizeof(L));
    L.items = d_items;
    L.n_items = n_blocks;
    L.threads = tn.threads;
    L.strip = tn.strip;
    L.mask_filters = F;
    L.total_units = nu * n_blocks;
    L.nf_max = std::max<uint32_t>(nf, 1);
    L.direct = 1;
    L.unit_counter = d_unit;
    L.surv = d_out;
    L.surv_n = d_count;
    L.surv_cap = out_cap;
    L.group_found = d_found;
    L.smem_bytes = sp.bytes;
    L.cnt_off = sp.cnt_off;
    L.queue_off = sp.queue_off;
    L.stage_off = sp.stage_off;
    launch_tables(L, I);
    if (L.total_units) {
        int grid = 0;
        if (int e = grid_for(layout, 0, I.W, F, tn, sp.bytes, L.total_units, &grid)) return e;
        int e = es_launch_scan(L, (int)layout, 0, I.W, grid, st);
        if (e) return cuda_fail((cudaError_t)e, "scan launch");
    }
    int e = es_launch_min(d_out, d_count, out_cap, d_items, 1, d_found, d_min, st);
    if (e) return cuda_fail((cudaError_t)e, "min launch");
    return ES_OK;
}
