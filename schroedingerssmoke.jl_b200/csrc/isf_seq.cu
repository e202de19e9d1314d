// Kernel sequences of the library's calls as graphs.
//
// On small grids a call is bound by its launches: about 1.9 us of host time
// each, against kernels of 1.5 to 3 us.  Jet steps of 16 kernels on 64x32x32,
// three simulations side by side, took 39 us each one by one and took 27.6 as
// graphs.  A sequence that a handle launches again and again (the same kernels
// in the same order) becomes an executable graph whose nodes are chained by
// programmatic edges, as the plain launches are.  Every call sets every node's
// shape and arguments (0.2 us each) and launches the graph (0.9 us): 13 kernels
// take 3.7 us of host time instead of 25 us, and 16.3 us back to back on one
// stream instead of 24.6 us.  Nothing is keyed by an address: another psi or
// particle buffer costs the same as the last one.
//
// A graph is built (about 100 us) on the fourth call of its sequence, so
// programs that make few calls never pay for it.
#include <string>
#include <utility>

#include "isf_handle.h"

namespace isf {
thread_local LaunchList* t_record = nullptr;
}

namespace isf_int {

namespace {

constexpr size_t kMaxSeqs = 16;       // sequences kept per handle
constexpr size_t kMaxNodes = 96;      // longer sequences are launched one by one
constexpr int kBuildAt = 4;           // the call of a sequence that builds its graph
// Grids up to which a sequence becomes a graph.  Where the GPU is the bound a
// graph gains nothing, and its start, which does not overlap the kernel before
// it, costs about 3 us: the driver loop's short sequences (flow, projection) on
// 128x64x64 ran 108 us one by one and 113 as graphs, on 100x50x50 103 and 107
// but 76 and 54 with three simulations side by side.  The fused step's one
// long sequence was no slower up to 160x80x80 (155 and 149 us) and equal on
// 256x128x128.
constexpr size_t kLongSeq = 8;
constexpr long long kShortCells = 300000, kLongCells = 1LL << 21;

void args_of(LaunchList& l, const LaunchList::Rec& r, std::vector<void*>& out) {
    out.resize(r.nargs);
    for (size_t i = 0; i < r.nargs; ++i) out[i] = l.bytes.data() + l.offs[r.arg0 + i];
}

// the launches one after another; bad: the one that failed
cudaError_t issue(LaunchList& l, cudaStream_t st, const LaunchList::Rec** bad = nullptr) {
    std::vector<void*> args;
    for (const LaunchList::Rec& r : l.recs) {
        args_of(l, r, args);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = r.grid;
        cfg.blockDim = r.block;
        cfg.dynamicSmemBytes = r.smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelExC(&cfg, r.func, args.data());
        if (e != cudaSuccess) {
            if (bad) *bad = &r;
            return e;
        }
    }
    return cudaSuccess;
}

void drop(isf_seq& s) {
    if (s.exec) cudaGraphExecDestroy(s.exec);
    if (s.graph) cudaGraphDestroy(s.graph);
    s.exec = nullptr;
    s.graph = nullptr;
    s.nodes.clear();
}

// the thread's capture mode for the length of a scope
struct CaptureMode {
    cudaStreamCaptureMode mode;
    explicit CaptureMode(cudaStreamCaptureMode m) : mode(m) { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~CaptureMode() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// the sequence's graph: a chain of kernel nodes, each allowed to start
// while the one before it drains
cudaError_t add_nodes(isf_seq& s, LaunchList& l) {
    std::vector<void*> args;
    cudaError_t e = cudaGraphCreate(&s.graph, 0);
    for (size_t i = 0; i < l.recs.size() && e == cudaSuccess; ++i) {
        const LaunchList::Rec& r = l.recs[i];
        args_of(l, r, args);
        cudaGraphNodeParams p = {};
        p.type = cudaGraphNodeTypeKernel;
        p.kernel.func = const_cast<void*>(r.func);
        p.kernel.gridDim = r.grid;
        p.kernel.blockDim = r.block;
        p.kernel.sharedMemBytes = (unsigned)r.smem;
        p.kernel.kernelParams = args.data();
        cudaGraphEdgeData edge = {};
        edge.from_port = cudaGraphKernelNodePortProgrammatic;
        edge.type = cudaGraphDependencyTypeProgrammatic;
        cudaGraphNode_t node;
        e = i ? cudaGraphAddNode_v2(&node, s.graph, &s.nodes.back(), &edge, 1, &p)
              : cudaGraphAddNode_v2(&node, s.graph, nullptr, nullptr, 0, &p);
        if (e == cudaSuccess) s.nodes.push_back(node);
    }
    return e == cudaSuccess ? cudaGraphInstantiate(&s.exec, s.graph, 0) : e;
}

// builds the graph, or leaves the sequence to plain launches for good
bool build(isf_seq& s, LaunchList& l) {
    // a capture elsewhere in the process is none of this graph's business
    CaptureMode relaxed(cudaStreamCaptureModeRelaxed);
    cudaError_t e;
    try {
        e = add_nodes(s, l);
    } catch (const std::bad_alloc&) {
        e = cudaErrorMemoryAllocation;
    }
    if (e == cudaSuccess) return true;
    cudaGetLastError();
    drop(s);
    s.failed = true;
    return false;
}

cudaError_t replay(isf_seq& s, LaunchList& l, cudaStream_t st) {
    std::vector<void*> args;
    for (size_t i = 0; i < l.recs.size(); ++i) {
        const LaunchList::Rec& r = l.recs[i];
        args_of(l, r, args);
        cudaKernelNodeParams p = {};
        p.func = const_cast<void*>(r.func);
        p.gridDim = r.grid;
        p.blockDim = r.block;
        p.sharedMemBytes = (unsigned)r.smem;
        p.kernelParams = args.data();
        const cudaError_t e = cudaGraphExecKernelNodeSetParams(s.exec, s.nodes[i], &p);
        if (e != cudaSuccess) return e;
    }
    return cudaGraphLaunch(s.exec, st);
}

// the handle's entry for the recorded kernels, or null when it has kMaxSeqs
// others (a handle's calls make fewer)
isf_seq* find(isf_handle* h) {
    const LaunchList& l = h->rec;
    for (isf_seq& s : h->seqs) {
        bool same = s.funcs.size() == l.recs.size();
        for (size_t i = 0; same && i < s.funcs.size(); ++i) same = s.funcs[i] == l.recs[i].func;
        if (same) return &s;
    }
    if (h->seqs.size() >= kMaxSeqs) return nullptr;
    isf_seq s;
    for (const LaunchList::Rec& r : l.recs) s.funcs.push_back(r.func);
    h->seqs.push_back(std::move(s));
    return &h->seqs.back();
}

}  // namespace

Sequence::Sequence(isf_handle* h, cudaStream_t st, const char* where)
    : h_(h), st_(st), where_(where), outer_(t_record), on_(!h->prof_on && !t_record) {
    if (!on_) return;
    h->rec.clear();
    t_record = &h->rec;
}

Sequence::~Sequence() {
    if (!on_) return;
    t_record = outer_;
    try {
        issue(h_->rec, st_);  // the call's own error is the one reported
    } catch (const std::bad_alloc&) {
    }
}

int Sequence::submit() {
    if (!on_) return ISF_OK;  // issued already, or part of an outer sequence
    t_record = outer_;
    on_ = false;
    try {
        return launch();
    } catch (const std::bad_alloc&) {
        return fail(h_, ISF_ERR_NOMEM, std::string(where_) + ": host allocation failed");
    }
}

int Sequence::launch() {
    LaunchList& l = h_->rec;
    if (l.recs.empty()) return ISF_OK;
    const size_t n = l.recs.size();
    if (n > 1 && n <= kMaxNodes && h_->g.N <= (n >= kLongSeq ? kLongCells : kShortCells)) {
        // a stream under capture takes the launches themselves
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        const bool free_stream = cudaStreamIsCapturing(st_, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
        if (!free_stream) cudaGetLastError();
        isf_seq* s = free_stream ? find(h_) : nullptr;
        if (s && s->seen < kBuildAt) ++s->seen;
        if (s && (s->exec || (s->seen == kBuildAt && !s->failed && build(*s, l)))) {
            const cudaError_t e = replay(*s, l, st_);
            if (e == cudaSuccess) return ISF_OK;
            // nothing of it was launched: the plain launches report what is wrong
            cudaGetLastError();
            cudaStreamSynchronize(st_);
            drop(*s);
            s->failed = true;
        }
    }
    const LaunchList::Rec* bad = nullptr;
    const cudaError_t e = issue(l, st_, &bad);
    if (e == cudaSuccess) return ISF_OK;
    return cuda_fail(h_, e, bad && bad->site ? l.names.data() + bad->site : where_);
}

bool seq_reserve(isf_handle* h) {
    try {
        h->rec.recs.reserve(32);
        h->rec.offs.reserve(64);
        h->rec.bytes.reserve(32 * 1024);
        h->rec.names.reserve(1024);
        return true;
    } catch (const std::bad_alloc&) {
        return false;
    }
}

void seq_free(isf_handle* h) {
    for (isf_seq& s : h->seqs) drop(s);
    h->seqs.clear();
}

}  // namespace isf_int
