// The engine's host code (csrc/llg_engine.cu and the planners) on a device that only keeps a record: device memory is the
// host's, a launch notes its kind and its stream, and any call can be made to fail.  Each scenario prints what went wrong
// and returns 1, or prints "ok".
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <random>
#include <set>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/llgpu.h"
#include "llg_internal.h"
#include "llg_launch.h"

namespace {

std::map<std::string, int> calls;     // by kind
std::map<std::string, int> fail_at;   // kind -> the call (from 1) that fails
// per stream: pieces of work issued and known to have ended; per event: its stream and how far that was; per stream: how
// far it has waited for others
std::map<void*, int> issued, ended;
std::map<void*, std::pair<void*, int>> recorded;
std::map<void*, std::map<void*, int>> waited;
size_t free_bytes = (size_t)200 << 30;
std::map<void*, size_t> live;
int malloc_limit = -1;                // pieces of 4 KB and more that are left (-1: any number)

cudaError_t call(const char* kind, cudaError_t error = cudaErrorUnknown) {
    const int k = ++calls[kind];
    const auto f = fail_at.find(kind);
    return f != fail_at.end() && f->second == k ? error : cudaSuccess;
}
cudaError_t work(const char* kind, cudaStream_t s) {
    const cudaError_t e = call(kind);
    if (e == cudaSuccess) ++issued[(void*)s];
    return e;
}

}  // namespace

// ---- the runtime ----
extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "planted"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { return *f = free_bytes, *t = (size_t)256 << 30, cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    const cudaError_t e = call("malloc", cudaErrorMemoryAllocation);
    if (malloc_limit >= 0 && n >= 4096 && --malloc_limit < 0) {
        malloc_limit = 0;
        return *p = nullptr, cudaErrorMemoryAllocation;
    }
    if (e != cudaSuccess || n > free_bytes) return *p = nullptr, cudaErrorMemoryAllocation;
    free_bytes -= n;
    *p = std::malloc(n < 64 ? 64 : n);
    live[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (p) free_bytes += live[p], live.erase(p);
    return std::free(p), cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = std::malloc(n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
static uintptr_t next_handle = 16;
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)(next_handle += 16), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)(next_handle += 16), cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    recorded[(void*)e] = {(void*)s, issued[(void*)s]};
    return call("event record");
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.f, cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    const cudaError_t rc = call("wait event");
    const auto at = recorded[(void*)e];
    if (rc == cudaSuccess) waited[(void*)s][at.first] = std::max(waited[(void*)s][at.first], at.second);
    return rc;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    ended[(void*)s] = issued[(void*)s];
    for (const auto& w : waited[(void*)s]) ended[w.first] = std::max(ended[w.first], w.second);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
    std::memset(p, v, n);
    return work("memset", s);
}
cudaError_t cudaMemcpyAsync(void* d, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    std::memmove(d, src, n);
    return work("copy", s);
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    return std::memset(a, 0, sizeof(*a)), a->type = cudaMemoryTypeUnregistered, cudaSuccess;
}
}

// ---- the kernels ----
namespace llg {
bool gate_block_eligible(int P, int n) { return (P == LLG_F64 || P == LLG_DF64) && n >= kBlockMinQubits; }
size_t gate_block_weight_bytes(int P) { return P == LLG_F64 ? 65792 : 57600; }
int64_t gate_block_launches() { return calls["block"]; }
cudaError_t launch_gate_block_weights(int, const BlockGate*, const BlockStep*, int, void*, cudaStream_t s, const double2*, const double2*,
                                      int, int, bool) {
    return work("weights", s);
}
cudaError_t launch_gate_block(int, void*, int, const BlockDesc&, const void*, bool, bool, int*, cudaStream_t s, double*) {
    return work("block", s);
}
size_t elem_bytes(int P) { return P == LLG_F32 ? 8 : 16; }
int tile_max_qubits(int P) { return P == LLG_F32 ? 14 : 13; }
cudaError_t launch_tile_pass(int, void*, int, const PassDesc&, const ExecOp*, const uint64_t*, int, int*, cudaStream_t s, double*) {
    return work("tile", s);
}
cudaError_t launch_exec_op(int, void*, int, const ExecOp&, cudaStream_t s) { return work("gate", s); }
cudaError_t launch_init_basis(int, void*, uint64_t, uint64_t, cudaStream_t s) { return work("init", s); }
cudaError_t launch_reduce_z(int, const void*, int, const ZTerms&, double*, unsigned*, const int*, Readout* host, cudaStream_t s) {
    std::memset(host, 0, sizeof(*host));
    host->red[0] = 1.0;
    return work("reduce", s);
}
}  // namespace llg

namespace {

llg_op op(int kind, int q0, int q1 = 0, double theta = 0.0) {
    llg_op o;
    std::memset(&o, 0, sizeof(o));
    o.kind = kind;
    o.q0 = q0;
    o.q1 = q1;
    o.theta = theta;
    o.param = -1;
    return o;
}

// rotations on every qubit and a brickwork of CNOTs
std::vector<llg_op> layered(int n, int layers) {
    std::mt19937 rng(7);
    std::uniform_real_distribution<double> angle(0.2, 3.0);
    std::vector<llg_op> q;
    for (int l = 0; l < layers; ++l) {
        for (int i = 0; i < n; ++i)
            for (int k : {LLG_OP_RX, LLG_OP_RY, LLG_OP_RZ}) q.push_back(op(k, i, 0, angle(rng)));
        for (int i = l % 2; i + 1 < n; i += 2) q.push_back(op(LLG_OP_CNOT, i, i + 1));
    }
    return q;
}

int fail(const char* what) {
    std::printf("%s\n", what);
    return 1;
}

bool idle() {
    for (const auto& p : issued)
        if (ended[p.first] < p.second) return false;
    return true;
}

// A call on the second stream fails: the flush reports it, and no work is left on either stream that may use the buffers that
// the next flush fills or that the end of the state frees.
int second_stream(const char* kind, int from, int count) {
    for (int at = from; at < from + count; ++at) {
        llg_state* st = nullptr;
        if (llg_create(14, LLG_F64, &st)) return fail("create");
        const std::vector<llg_op> q = layered(14, 40);
        if (llg_apply_ops(st, q.data(), (int)q.size())) return fail("apply");
        calls.clear();
        fail_at = {{kind, at}};
        if (llg_flush(st) == LLG_OK) return fail("the failing call was not reported");
        if (!calls["weights"]) return fail("the list did not run in blocks");
        if (!idle()) return fail("work in flight after a failed flush");
        fail_at.clear();
        if (llg_apply_ops(st, q.data(), (int)q.size()) || llg_sync(st)) return fail("the next flush");
        llg_destroy(st);
        if (!idle()) return fail("work in flight at the end of the state");
    }
    return 0;
}

std::vector<llg_op> read_ops(const char* path) {
    std::vector<llg_op> q;
    if (FILE* f = std::fopen(path, "rb")) {
        llg_op o;
        while (std::fread(&o, sizeof(o), 1, f) == 1) q.push_back(o);
        std::fclose(f);
    }
    return q;
}

// The block plan of the gate records in a file, up to `blocks` blocks, and the gates that are left then: counts, steps, gates,
// records to another file.
int plan(int n, int blocks, const char* path, const char* out) {
    const std::vector<llg_op> q = read_ops(path);
    llg::BlockPlanner p(n, q.data(), (int)q.size());
    p.advance(blocks);
    p.mark();
    const size_t steps = p.plan.steps.size(), gates = p.plan.gates.size();
    p.advance(3);  // not marked: its gates are left
    const std::vector<llg_op> left = p.rest(q.data(), (int)q.size());
    const long long counts[3] = {(long long)steps, (long long)gates, (long long)left.size()};
    FILE* f = std::fopen(out, "wb");
    if (!f) return fail("open");
    std::fwrite(counts, sizeof(counts), 1, f);
    std::fwrite(p.plan.steps.data(), sizeof(llg::BlockStep), steps, f);
    std::fwrite(p.plan.gates.data(), sizeof(llg::BlockGate), gates, f);
    std::fwrite(left.data(), sizeof(llg_op), left.size(), f);
    std::fclose(f);
    return 0;
}

// The launches of one flush of the gate records in a file, from |0..0>.
int flush(int n, int precision, const char* path) {
    const std::vector<llg_op> q = read_ops(path);
    llg_state* st = nullptr;
    if (llg_create(n, precision, &st) || llg_apply_ops(st, q.data(), (int)q.size())) return fail("create");
    calls.clear();
    if (llg_flush(st)) return fail("flush");
    std::printf("%d %d %d\n", calls["block"], calls["tile"], calls["gate"]);
    llg_destroy(st);
    return 0;
}

// A long list with room for `more` pieces of memory only: the weights' parts take turns, and no work waits for room.
int little_room(int more) {
    llg_state* st = nullptr;
    const std::vector<llg_op> q = layered(14, 200);  // some 400 blocks in 26 groups
    if (llg_create(14, LLG_F64, &st) || llg_set_fusion(st, LLG_FUSE_TILE, 12)) return fail("create");
    if (llg_apply_ops(st, q.data(), (int)q.size()) || llg_sync(st)) return fail("tile passes");  // their buffers are kept
    if (llg_set_fusion(st, LLG_FUSE_TILE, 0) || llg_apply_ops(st, q.data(), (int)q.size())) return fail("apply");
    calls.clear();
    malloc_limit = more;
    if (llg_sync(st)) return fail("flush");
    const int first = calls["block"];
    // one piece for the plan, one for the first group's weights
    if ((first > 0) != (more >= 2)) return fail(more >= 2 ? "blocks had room" : "blocks had no room");
    if (first == 0 && calls["tile"] == 0) return fail("neither form ran");
    malloc_limit = -1;
    if (llg_apply_ops(st, q.data(), (int)q.size()) || llg_sync(st)) return fail("the next flush");
    if (calls["block"] <= first) return fail("blocks have room again");
    llg_destroy(st);
    if (!idle() || !live.empty()) return fail("memory or work left at the end of the state");
    return 0;
}

}  // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    int rc = 2;
    if (what == "weights") rc = second_stream("weights", 2, 3);
    if (what == "copy") rc = second_stream("copy", 2, 3);
    if (what == "record") rc = second_stream("event record", 1, 4);
    if (what == "wait") rc = second_stream("wait event", 1, 2);
    if (what == "block") rc = second_stream("block", 20, 20);
    if (what == "room" && argc == 3) rc = little_room(std::atoi(argv[2]));
    if (what == "plan" && argc == 6) rc = plan(std::atoi(argv[2]), std::atoi(argv[3]), argv[4], argv[5]);
    if (what == "flush" && argc == 5) return flush(std::atoi(argv[2]), std::atoi(argv[3]), argv[4]);
    if (!rc) std::printf("ok\n");
    return rc;
}
