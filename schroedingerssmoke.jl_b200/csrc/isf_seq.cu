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
// A graph costs 60 to 85 us of host time to build and 50 to give back, and saves
// 5 to 15 us a call.  It is built on the 16th call of its sequence, when those
// before would have paid for it; a handle that makes fewer never pays, and its
// calls launch their kernels as they come, as if there were no sequences
// (recording first makes a single call 1 to 2 us longer).
#include <string>
#include <utility>

#include "isf_handle.h"

namespace isf {
thread_local LaunchList* t_record = nullptr;
}

namespace isf_int {

namespace {

constexpr size_t kMaxSeqs = 16;       // sequences kept per handle
constexpr size_t kMaxNodes = 32;      // longer sequences are launched one by one (a step has up to 17)
constexpr int kBuildAt = 16;          // the call of a sequence that builds its graph

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

// the handle's entry for the kernels in h->rec, or -1 when it has kMaxSeqs
// others (a handle's calls make fewer)
int find(isf_handle* h) {
    const LaunchList& l = h->rec;
    for (size_t k = 0; k < h->seqs.size(); ++k) {
        const isf_seq& s = h->seqs[k];
        bool same = s.funcs.size() == l.recs.size();
        for (size_t i = 0; same && i < s.funcs.size(); ++i) same = s.funcs[i] == l.recs[i].func;
        if (same) return (int)k;
    }
    if (h->seqs.size() >= kMaxSeqs) return -1;
    isf_seq s;
    for (const LaunchList::Rec& r : l.recs) s.funcs.push_back(r.func);
    h->seqs.push_back(std::move(s));
    return (int)h->seqs.size() - 1;
}

// the handle's note of a kind of call, or null when it has no room
isf_handle::SeqSite* site_of(isf_handle* h, const char* where) {
    for (isf_handle::SeqSite& s : h->seq_sites) {
        if (!s.where) s = {where, -1};
        if (s.where == where) return &s;
    }
    return nullptr;
}

// does the next call of the sequence go through a graph?
bool ready(const isf_seq& s) { return s.exec || (!s.failed && s.seen >= kBuildAt - 1); }

}  // namespace

Sequence::Sequence(isf_handle* h, cudaStream_t st, const char* where, long long max_cells)
    : h_(h), st_(st), where_(where), outer_(t_record), on_(!h->prof_on && !t_record && h->g.N <= max_cells) {
    if (!on_) return;
    h->rec.clear();
    h->rec.hold = false;
    site_ = site_of(h, where);
    if (site_ && site_->last >= 0 && ready(h->seqs[site_->last])) {
        // a stream under capture takes the launches themselves
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) cudaGetLastError();
        else h->rec.hold = cap == cudaStreamCaptureStatusNone;
    }
    t_record = &h->rec;
}

Sequence::~Sequence() {
    if (!on_) return;
    t_record = outer_;
    if (!h_->rec.hold) return;
    try {
        issue(h_->rec, st_);  // the call's own error is the one reported
    } catch (const std::bad_alloc&) {
    }
    h_->rec.hold = false;
}

int Sequence::submit() {
    if (!on_) return ISF_OK;  // issued already, or part of an outer sequence
    t_record = outer_;
    on_ = false;
    const bool hold = h_->rec.hold;
    int rc;
    try {
        rc = launch();
    } catch (const std::bad_alloc&) {
        rc = hold ? fail(h_, ISF_ERR_NOMEM, std::string(where_) + ": host allocation failed") : ISF_OK;
    }
    h_->rec.hold = false;
    return rc;
}

int Sequence::launch() {
    LaunchList& l = h_->rec;
    const size_t n = l.recs.size();
    if (n == 0) return ISF_OK;
    const int k = n > 1 && n <= kMaxNodes && !l.over ? find(h_) : -1;
    if (site_) site_->last = k;
    if (k >= 0 && l.hold) {
        isf_seq& s = h_->seqs[k];
        const bool was_failed = s.failed;
        if (s.exec || (ready(s) && build(s, l))) {
            if (replay(s, l, st_) == cudaSuccess) {
                ++h_->graph_launches;
                return ISF_OK;
            }
            // nothing of it was launched: the plain launches report what is wrong
            cudaGetLastError();
            cudaStreamSynchronize(st_);
            drop(s);
            s.failed = true;
        }
        if (s.failed && !was_failed) ++h_->graph_failures;
    }
    if (k >= 0 && h_->seqs[k].seen < kBuildAt - 1) ++h_->seqs[k].seen;
    if (!l.hold) return ISF_OK;  // launched as they came
    const LaunchList::Rec* bad = nullptr;
    const cudaError_t e = issue(l, st_, &bad);
    if (e == cudaSuccess) return ISF_OK;
    return cuda_fail(h_, e, bad && bad->site ? bad->site : where_);
}

bool seq_reserve(isf_handle* h) {
    try {
        h->rec.recs.reserve(kMaxNodes);
        h->rec.offs.reserve(64);
        h->rec.bytes.reserve(32 * 1024);
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
