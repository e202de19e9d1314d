// Runs the kernel sequences of csrc/isf_seq.cu against the CUDA runtime of
// seq_runtime.cpp, without a GPU: what is launched, in which form and in which
// order, is printed, and a launch or a host allocation can be made to fail.
// Built and driven by test_sequences_cpu.py.
#include <cstdio>
#include <cstdlib>
#include <string>

#include "isf_handle.h"

// the runtime's switches (seq_runtime.cpp)
extern int g_fail_launch;   // the kernel launch (by number) that fails
extern bool g_fail_graph;   // cudaGraphLaunch fails
extern long g_fail_new;     // the host allocation (counted from arming) that fails
extern int g_mode;          // capture interaction mode of the thread
extern int g_graphs;        // live graphs

// ------------------------------------------------- the rest of the library
namespace isf_int {
int fail(isf_handle* h, int code, const std::string& msg) {
    h->err = msg;
    return code;
}
int cuda_fail(isf_handle* h, cudaError_t, const char* where) {
    h->err = where;
    return ISF_ERR_CUDA;
}
int prof_begin(isf_handle*, const char*, cudaStream_t) { return -1; }
void prof_end(isf_handle*, int, cudaStream_t) {}
}  // namespace isf_int

using namespace isf;
using namespace isf_int;

__global__ void ka(int) {}
__global__ void kb(int) {}
__global__ void kc(int) {}

// a call of three kernels without kernel `skip`, the host failing before kernel
// `stop` (3: not at all)
static int call(isf_handle* h, int tag, int stop = 3, int skip = -1) {
    Sequence seq(h, nullptr, "call", 4096);
    void (*const k[3])(int) = {ka, kb, kc};
    const char* const site[3] = {"pass a", "pass b", "pass c"};
    for (int i = 0; i < 3; ++i) {
        if (i == stop) return fail(h, ISF_ERR_INVALID, "stopped");
        if (i == skip) continue;
        ISF_LAUNCH(h, launch_pdl(k[i], dim3(1), dim3(32), 0, nullptr, 10 * tag + i), site[i]);
    }
    return seq.submit();
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const int n = argc > 2 ? std::atoi(argv[2]) : 0;
    const int before = argc > 3 ? std::atoi(argv[3]) : 0;  // calls before the one that matters
    isf_handle h;
    h.g.N = what == "large" ? 4097 : 4096;
    if (!seq_reserve(&h)) return 1;
    for (int i = 1; i <= before; ++i)
        if (call(&h, i)) return 1;
    const int tag = before + 1;
    if (what == "repeat" || what == "large") {  // n calls
        for (int i = 0; i < n; ++i)
            if (call(&h, tag + i)) return 1;
    } else if (what == "other") {  // n calls of other kernels
        for (int i = 0; i < n; ++i)
            if (call(&h, tag + i, 3, 1)) return 1;
    } else if (what == "stop") {  // the host fails after n kernels
        const int rc = call(&h, tag, n);
        std::printf("rc %d %s recording %d\n", rc, h.err.c_str(), t_record != nullptr);
    } else if (what == "launch") {  // kernel n cannot be launched, nor can the graph
        g_fail_launch = 3 * before + n;
        g_fail_graph = true;
        if (before > 15) g_fail_launch = 3 * 15 + n;
        const int rc = call(&h, tag);
        std::printf("rc %d %s\n", rc, h.err.c_str());
    } else if (what == "build") {  // host allocation n of the call fails
        g_fail_new = n;
        const int rc = call(&h, tag);
        const bool failed = g_fail_new < 0;
        g_fail_new = -1;
        std::printf("rc %d mode %d\n", rc, g_mode);
        if (call(&h, tag + 1)) return 1;
        if (!failed) std::printf("all\n");
    } else if (what == "reserve") {  // host allocation n of the handle's fails
        isf_handle other;
        g_fail_new = n;
        const bool ok = seq_reserve(&other);
        std::printf("%s\n", ok ? (g_fail_new < 0 ? "missed" : "all") : "no room");
        g_fail_new = -1;
    } else {
        return 2;
    }
    seq_free(&h);
    std::printf("mode %d graphs %d\n", g_mode, g_graphs);
    return 0;
}
