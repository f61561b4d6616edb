#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <vector>
#include <map>
#include <mutex>
#include <tuple>
#include <unordered_map>
#include <utility>

#include "runtime.hpp"

namespace mops_b200 {

[[noreturn]] void throw_cuda(cudaError_t err, const char* what, const char* file, int line) {
    // Clear the (non-sticky) error so that the next call starts clean.
    (void)cudaGetLastError();
    throw std::runtime_error(
        std::string("CUDA error: ") + cudaGetErrorString(err) + " in `" + what + "` at " + file +
        ":" + std::to_string(line));
}

// What a thread keeps for a (device, stream): calls on one stream run in order, so a call's status
// words and workspace cannot be overwritten before its own kernels are done with them, and calls on
// different streams (which may overlap) never share them. Status words are never freed (kernels of
// captured graphs hold their address) but handed on, with the workspace, to later streams.
struct StreamState {
    Status status{};
    unsigned char* workspace = nullptr;
    size_t size = 0, used = 0;
    size_t wanted = 0; // by the previous call
    bool pending = false; // a call may still be running (it did not wait, or ended with an exception)
    bool captured = false; // a graph holds the address of the status words
    uint64_t last_call = 0;
};

namespace {

// Lets this thread wait and free while another thread captures a graph.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
};

constexpr size_t kMostWorkspace = 4 << 20; // bytes per (thread, device, stream)
constexpr int kMostWorkspaces = 16;        // per thread
constexpr size_t kMostStreams = 64;        // per thread, before states of old streams are handed on

struct ThreadState {
    cudaStream_t stream = nullptr;
    bool wait = true;
    uint32_t epoch = 0;
    // by device and stream id: a handle may come back for another stream, an id does not
    std::map<std::pair<int, unsigned long long>, StreamState> streams;
    std::vector<std::pair<int, StreamState>> spare; // (device, state) of streams that have gone
    uint64_t calls = 0;
    std::pair<int, unsigned long long> last_key{-1, 0};
    StreamState* last = nullptr; // of the previous call
    int workspaces = 0;
    std::string kernels; // main kernels dispatched by the current / last call

    // The thread is gone, its kernels may not be: cudaFree does not wait for the users of memory from a
    // stream-ordered pool. (Where the device cannot be waited for, the workspace is left behind.)
    ~ThreadState() {
        int device = 0;
        if (workspaces == 0 || cudaGetDevice(&device) != cudaSuccess) return;
        const RelaxedCapture relaxed;
        auto give_back = [](int on, const StreamState& s) {
            if (s.workspace == nullptr) return;
            if (!s.pending || (cudaSetDevice(on) == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess))
                (void)cudaFree(s.workspace);
            (void)cudaGetLastError();
        };
        for (auto& s : streams) give_back(s.first.first, s.second);
        for (auto& s : spare) give_back(s.first, s.second);
        (void)cudaSetDevice(device);
    }
};

thread_local ThreadState g_thread;

struct DeviceInfo {
    int sms = 0;
    int smem = 0;
};
std::mutex g_info_mutex;
std::unordered_map<int, DeviceInfo> g_info;

const DeviceInfo& device_info(int device) {
    std::lock_guard<std::mutex> lock(g_info_mutex);
    auto it = g_info.find(device);
    if (it == g_info.end()) {
        DeviceInfo info;
        MOPS_CUDA_OK(cudaDeviceGetAttribute(&info.sms, cudaDevAttrMultiProcessorCount, device));
        MOPS_CUDA_OK(
            cudaDeviceGetAttribute(&info.smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
        it = g_info.emplace(device, info).first;
    }
    return it->second;
}

} // namespace

int sm_count(int device) { return device_info(device).sms; }
int max_optin_smem(int device) { return device_info(device).smem; }

void set_stream(void* stream) { g_thread.stream = static_cast<cudaStream_t>(stream); }
void* get_stream() { return g_thread.stream; }
void set_wait(bool wait) { g_thread.wait = wait; }
bool get_wait() { return g_thread.wait; }

namespace {
// Zeros device words before any kernel can use them. On a stream of its own and waited for: a memset on
// the legacy default stream is in order with neither the host nor a non-blocking stream, and could
// wipe out what the first call's kernels have written.
void zero_words(uint32_t* dev, int words) {
    cudaStream_t stream = nullptr;
    MOPS_CUDA_OK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    cudaError_t err = cudaMemsetAsync(dev, 0, words * sizeof(uint32_t), stream);
    if (err == cudaSuccess) err = cudaStreamSynchronize(stream);
    (void)cudaStreamDestroy(stream);
    MOPS_CUDA_OK(err);
}

// Ids of streams never come back, so a program that makes a stream per step would leave a state behind
// each time. At kMostStreams the older half of them (but for graphs') goes to `spare`, once the device
// has been waited for if any of their calls may still run: one wait in kMostStreams / 2 new streams.
// Where it cannot be waited for, the states stay.
void retire_streams(int device) {
    std::vector<std::pair<uint64_t, std::pair<int, unsigned long long>>> old;
    for (const auto& s : g_thread.streams)
        if (s.first.first == device && !s.second.captured) old.push_back({s.second.last_call, s.first});
    std::sort(old.begin(), old.end());
    old.resize(std::min(old.size(), kMostStreams / 2));
    const RelaxedCapture relaxed;
    bool pending = false;
    for (const auto& o : old) pending |= g_thread.streams[o.second].pending;
    if (old.empty() || (pending && cudaDeviceSynchronize() != cudaSuccess)) {
        (void)cudaGetLastError();
        return;
    }
    g_thread.last = nullptr;
    for (const auto& o : old) {
        StreamState& state = g_thread.streams[o.second];
        state.pending = false;
        g_thread.spare.push_back({device, state});
        g_thread.streams.erase(o.second);
    }
}

StreamState& state_of(const std::pair<int, unsigned long long>& key, bool capturing) {
    auto it = g_thread.streams.find(key);
    if (it != g_thread.streams.end()) return it->second;
    if (g_thread.streams.size() >= kMostStreams && !capturing) retire_streams(key.first);
    // (a spare one with a workspace rather than one without)
    auto spare = g_thread.spare.end();
    for (auto s = g_thread.spare.begin(); s != g_thread.spare.end(); ++s)
        if (s->first == key.first && (spare == g_thread.spare.end() || s->second.workspace != nullptr)) spare = s;
    StreamState state{};
    if (spare != g_thread.spare.end()) {
        state = spare->second;
        g_thread.spare.erase(spare);
    } else {
        void* host = nullptr;
        // (with unified addressing the host pointer is the device-visible one)
        MOPS_CUDA_OK(cudaHostAlloc(&host, kStatusWords * sizeof(uint32_t),
                                   cudaHostAllocMapped | cudaHostAllocPortable));
        for (int i = 0; i < kStatusWords; i++) static_cast<volatile uint32_t*>(host)[i] = 0;
        state.status.host = static_cast<uint32_t*>(host);
        MOPS_CUDA_OK(cudaMalloc(reinterpret_cast<void**>(&state.status.dev), kStatusWords * sizeof(uint32_t)));
        zero_words(state.status.dev, kStatusWords);
    }
    return g_thread.streams.emplace(key, state).first->second;
}
} // namespace

Call begin_call() {
    Call call;
    MOPS_CUDA_OK(cudaGetDevice(&call.device));
    call.stream = g_thread.stream;
    call.wait = g_thread.wait;

    g_thread.kernels.clear();
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(call.stream, &capture) != cudaSuccess) (void)cudaGetLastError();
    call.capturing = capture != cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    MOPS_CUDA_OK(cudaStreamGetId(call.stream, &id));
    const auto key = std::make_pair(call.device, id);
    if (g_thread.last == nullptr || key != g_thread.last_key) {
        g_thread.last = &state_of(key, call.capturing);
        g_thread.last_key = key;
    }
    call.state = g_thread.last;
    call.state->used = 0;
    call.state->pending = true;
    call.state->captured |= call.capturing;
    call.state->last_call = ++g_thread.calls;
    call.status = call.state->status;
    g_thread.epoch += 1;
    if (g_thread.epoch == 0) g_thread.epoch = 1;
    call.status.epoch = g_thread.epoch;
    return call;
}

void note_kernel(const std::string& name) {
    if (!g_thread.kernels.empty()) g_thread.kernels += "; ";
    g_thread.kernels += name;
}
void note_kernel_f(const char* format, ...) {
    char text[160];
    va_list args;
    va_start(args, format);
    vsnprintf(text, sizeof(text), format, args);
    va_end(args);
    note_kernel(text);
}
const char* last_kernels() { return g_thread.kernels.c_str(); }

void wait_stream(const Call& call) { MOPS_CUDA_OK(cudaStreamSynchronize(call.stream)); }

bool host_saw_unsorted(const Call& call) {
    return static_cast<volatile uint32_t*>(call.status.host)[kUnsortedEpoch] == call.status.epoch;
}

void end_call(const Call& call, const char* operation, const char* const* index_names,
              int n_index_names) {
    MOPS_CUDA_OK(cudaGetLastError());
    if (!call.wait) return;
    MOPS_CUDA_OK(cudaStreamSynchronize(call.stream));
    call.state->pending = false;
    volatile uint32_t* host = call.status.host;
    if (host[kStalled] == call.status.epoch)
        throw std::runtime_error(std::string("internal error in operation ") + operation +
                                 ": a kernel gave up waiting for an asynchronous copy; the "
                                 "results of this call are incomplete");
    std::string names;
    for (int i = 0; i < n_index_names && i < kMaxIndexArrays; i++) {
        if (host[kBadIndex0 + i] == call.status.epoch) {
            if (!names.empty()) names += ", ";
            names += index_names[i];
        }
    }
    if (!names.empty()) {
        throw std::runtime_error(
            "Index array " + names + " in operation " + operation +
            " contains negative or too large elements; this would cause out-of-bounds accesses");
    }
}

namespace {
// One stream-ordered pool per device that keeps freed blocks instead of returning them to the
// driver at the next synchronisation (the default pool's behaviour, which would make every
// call pay for mapping its scratch memory again).
std::mutex g_pool_mutex;
std::unordered_map<int, cudaMemPool_t> g_pools;

cudaMemPool_t scratch_pool(int device) {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    auto it = g_pools.find(device);
    if (it == g_pools.end()) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        MOPS_CUDA_OK(cudaMemPoolCreate(&pool, &props));
        uint64_t keep = UINT64_MAX;
        MOPS_CUDA_OK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        it = g_pools.emplace(device, pool).first;
    }
    return it->second;
}
} // namespace

// ---- plans
class TablePlan {
  public:
    struct Entry {
        TableKey key;
        int device;
        void* ptr;
        size_t bytes;
        bool ready;  // built and committed
        bool usable; // false: the index was unsorted or held bad values (rebuild per call)
    };
    std::mutex mutex;
    std::vector<Entry> entries;
};

namespace {
thread_local TablePlan* g_bound_plan = nullptr;
bool same_key(const TableKey& a, const TableKey& b) { return std::memcmp(&a, &b, sizeof(TableKey)) == 0; }
} // namespace

TablePlan* plan_create() { return new TablePlan(); }

void plan_destroy(TablePlan* plan) {
    if (plan == nullptr) return;
    if (g_bound_plan == plan) g_bound_plan = nullptr;
    for (auto& e : plan->entries) {
        if (e.ptr != nullptr) {
            int previous = 0;
            if (cudaGetDevice(&previous) == cudaSuccess && cudaSetDevice(e.device) == cudaSuccess) {
                (void)cudaFree(e.ptr);
                (void)cudaSetDevice(previous);
            }
        }
    }
    delete plan;
}

void plan_bind(TablePlan* plan) { g_bound_plan = plan; }
TablePlan* plan_bound() { return g_bound_plan; }

int plan_table_count(const TablePlan* plan) {
    if (plan == nullptr) return 0;
    std::lock_guard<std::mutex> lock(const_cast<TablePlan*>(plan)->mutex);
    int n = 0;
    for (const auto& e : plan->entries) n += e.ready && e.usable ? 1 : 0;
    return n;
}

TableRef acquire_table(const Call& call, const TableKey& key_in, size_t bytes) {
    TableRef ref{nullptr, true, false, false, -1};
    TablePlan* plan = g_bound_plan;
    if (plan != nullptr) {
        TableKey key;
        std::memset(&key, 0, sizeof(key)); // padding bytes take part in the comparison
        key.kind = key_in.kind;
        key.scalar_bytes = key_in.scalar_bytes;
        for (int i = 0; i < 5; i++) key.ptr[i] = key_in.ptr[i];
        for (int i = 0; i < 10; i++) key.n[i] = key_in.n[i];
        std::lock_guard<std::mutex> lock(plan->mutex);
        for (size_t i = 0; i < plan->entries.size(); i++) {
            TablePlan::Entry& e = plan->entries[i];
            if (e.device != call.device || !same_key(e.key, key)) continue;
            if (e.ready && e.usable) {
                ref.ptr = e.ptr;
                ref.fresh = false;
                ref.owned_by_plan = true;
                ref.sorted = true;
                ref.slot = static_cast<int>(i);
                return ref;
            }
            // known to be unusable (or being built by another thread): per-call scratch
            ref.ptr = scratch_alloc(call, bytes);
            return ref;
        }
        TablePlan::Entry e{};
        e.key = key;
        e.device = call.device;
        e.bytes = bytes;
        e.ready = false;
        e.usable = false;
        // plain cudaMalloc: the table outlives the call and is used from any stream
        MOPS_CUDA_OK(cudaMalloc(&e.ptr, bytes > 0 ? bytes : 1));
        plan->entries.push_back(e);
        ref.ptr = e.ptr;
        ref.owned_by_plan = true;
        ref.slot = static_cast<int>(plan->entries.size() - 1);
        return ref;
    }
    ref.ptr = scratch_alloc(call, bytes);
    return ref;
}

void commit_table(const Call& call, TableRef& ref) {
    if (!ref.owned_by_plan || !ref.fresh) return;
    TablePlan* plan = g_bound_plan;
    // The table must be complete before another stream may use it, and what its builder
    // reported decides whether it can be kept.
    MOPS_CUDA_OK(cudaStreamSynchronize(call.stream));
    volatile uint32_t* host = call.status.host;
    bool clean = true;
    for (int w = 0; w < kStatusWords; w++) clean = clean && host[w] != call.status.epoch;
    ref.sorted = clean;
    if (plan == nullptr) return;
    std::lock_guard<std::mutex> lock(plan->mutex);
    if (ref.slot >= 0 && ref.slot < static_cast<int>(plan->entries.size())) {
        plan->entries[ref.slot].ready = true;
        plan->entries[ref.slot].usable = clean;
    }
}

void release_table(const Call& call, const TableRef& ref) {
    if (!ref.owned_by_plan) scratch_free(call, ref.ptr);
}

void* scratch_alloc(const Call& call, size_t bytes) {
    StreamState& w = *call.state;
    bytes = (bytes + 255) / 256 * 256;
    if (bytes <= kMostWorkspace) {
        if (!call.capturing) {
            if (w.used == 0 && w.size < w.wanted) { // grow between calls, in stream order
                if (w.workspace != nullptr) {
                    MOPS_CUDA_OK(cudaFreeAsync(w.workspace, call.stream));
                    w.workspace = nullptr;
                    w.size = 0;
                    g_thread.workspaces--;
                }
                if (g_thread.workspaces < kMostWorkspaces) {
                    void* ptr = nullptr;
                    MOPS_CUDA_OK(cudaMallocFromPoolAsync(&ptr, w.wanted, scratch_pool(call.device), call.stream));
                    w.workspace = static_cast<unsigned char*>(ptr);
                    w.size = w.wanted;
                    g_thread.workspaces++;
                }
            }
            if (w.used + bytes <= w.size) {
                void* ptr = w.workspace + w.used;
                w.used += bytes;
                return ptr;
            }
            // not now: remember for the next call
            size_t want = w.used + bytes;
            want = want + want / 2 < kMostWorkspace ? want + want / 2 : kMostWorkspace;
            if (want > w.wanted) w.wanted = want;
        }
    }
    void* ptr = nullptr;
    MOPS_CUDA_OK(cudaMallocFromPoolAsync(&ptr, bytes, scratch_pool(call.device), call.stream));
    return ptr;
}

void scratch_free(const Call& call, void* ptr) {
    const unsigned char* p = static_cast<unsigned char*>(ptr);
    const StreamState& w = *call.state;
    if (p == nullptr || (w.workspace != nullptr && p >= w.workspace && p < w.workspace + w.size)) return;
    MOPS_CUDA_OK(cudaFreeAsync(ptr, call.stream));
}

// ---- launch settings
namespace {
std::mutex g_kernel_mutex;
std::map<std::pair<const void*, int>, size_t> g_kernel_smem;
std::map<std::tuple<const void*, int, int, size_t>, int> g_kernel_blocks;
} // namespace

void allow_dynamic_smem(const void* kernel, int device, size_t smem) {
    if (smem <= 48 * 1024) return; // allowed as it is
    std::lock_guard<std::mutex> lock(g_kernel_mutex);
    size_t& allowed = g_kernel_smem[{kernel, device}];
    if (smem <= allowed) return;
    MOPS_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(smem)));
    allowed = smem;
}

int resident_blocks(const void* kernel, int device, int threads, size_t smem) {
    allow_dynamic_smem(kernel, device, smem);
    std::lock_guard<std::mutex> lock(g_kernel_mutex);
    int& blocks = g_kernel_blocks[{kernel, device, threads, smem}];
    if (blocks == 0) {
        MOPS_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, threads, smem));
        if (blocks < 1) blocks = 1;
    }
    return blocks;
}

} // namespace mops_b200
