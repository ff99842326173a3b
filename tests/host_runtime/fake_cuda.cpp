#include "fake_cuda.h"

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <set>
#include <vector>

#include <cuda_runtime.h>

#include "sgl.h"
#include "sgl_internal.h"

namespace fake {
long unordered, overwritten, device_calls, streams_destroyed_twice, foreign_streams_destroyed;
size_t live, peak;
bool auto_progress;
std::string fail_on;

using Clock = std::map<const void *, long>; // per stream: operations known to be before

struct Event;
struct Op {
    enum Kind { kWork, kCopy, kWait } kind;
    void *dst = nullptr;
    const void *src = nullptr;
    size_t n = 0;
    uint64_t hash = 0;
    const void *other = nullptr; // kWait: that stream, up to `upto`
    long upto = 0;
};
struct Stream {
    std::deque<Op> ops;
    long enqueued = 0, done = 0; // operations so far
    Clock clock;
    bool by_test = false, capturing = false;
};
struct Event {
    const void *stream = nullptr;
    long at = 0;
    Clock clock;
};

static std::recursive_mutex mu;
static std::map<const void *, Stream> streams; // (nullptr: the legacy default stream)
static std::set<const void *> gone;
static Clock host;
static std::map<void *, size_t> device, pinned;
static const void *last_stream;
static long last_at;
static bool any_work;

static uint64_t hash_of(const void *p, size_t n)
{
    uint64_t h = 1469598103934665603ull;
    for (size_t i = 0; i < n; i++)
        h = (h ^ ((const uint8_t *)p)[i]) * 1099511628211ull;
    return h;
}
static bool is_pinned(const void *p)
{
    auto it = pinned.upper_bound((void *)p);
    return it != pinned.begin() && (const uint8_t *)p < (const uint8_t *)(--it)->first + it->second;
}
static void merge(Clock &a, const Clock &b)
{
    for (auto &x : b)
        a[x.first] = std::max(a[x.first], x.second);
}
static void drain(const void *s, long upto)
{
    Stream &st = streams[s];
    while (st.done < upto && !st.ops.empty()) {
        Op op = st.ops.front();
        st.ops.pop_front();
        st.done++;
        if (op.kind == Op::kWait)
            drain(op.other, op.upto);
        if (op.kind == Op::kCopy) {
            if (hash_of(op.src, op.n) != op.hash)
                overwritten++;
            memcpy(op.dst, op.src, op.n);
        }
    }
}
static void host_waits(const void *s, long upto, const Clock &c)
{
    drain(s, upto);
    merge(host, c);
}
void drain_all()
{
    std::lock_guard<std::recursive_mutex> g(mu);
    for (auto &s : streams)
        host_waits(s.first, s.second.enqueued, s.second.clock);
}
// Enqueues an operation; `work` is checked against the work before it.
static void enqueue(const void *s, const Op &op, bool work)
{
    Stream &st = streams[s];
    if (st.capturing)
        return;
    merge(st.clock, host);
    if (work) {
        device_calls++;
        if (any_work && last_stream != s && st.clock[last_stream] < last_at)
            unordered++;
    }
    st.ops.push_back(op);
    st.clock[s] = ++st.enqueued;
    if (work) {
        any_work = true;
        last_stream = s;
        last_at = st.enqueued;
    }
}
static bool fails(const char *what) { return fail_on == what; }
static cudaError_t launch(const char *what, cudaStream_t st)
{
    std::lock_guard<std::recursive_mutex> g(mu);
    if (fails(what))
        return cudaErrorLaunchFailure;
    enqueue(st, Op{Op::kWork}, true);
    return cudaSuccess;
}
} // namespace fake

using namespace fake;
#define LOCK std::lock_guard<std::recursive_mutex> g(mu)

extern "C" {
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMalloc(void **p, size_t n)
{
    LOCK;
    device_calls++;
    *p = aligned_alloc(256, (n + 255) / 256 * 256);
    memset(*p, 0, n);
    device[*p] = n;
    live += n;
    peak = std::max(peak, live);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    LOCK;
    drain_all(); // (waits for the device)
    if (p) {
        live -= device[p];
        device.erase(p);
        free(p);
    }
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    LOCK;
    *p = calloc(1, n);
    pinned[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p)
{
    LOCK;
    pinned.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    LOCK;
    *s = (cudaStream_t) new int(0);
    streams[*s];
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    LOCK;
    if (!gone.insert(s).second)
        streams_destroyed_twice++;
    else if (streams[s].by_test)
        foreign_streams_destroyed++;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    LOCK;
    host_waits(s, streams[s].enqueued, streams[s].clock);
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize()
{
    drain_all();
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, enum cudaStreamCaptureStatus *c)
{
    return *c = cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
    LOCK;
    Event &ev = *(Event *)e;
    Op op{Op::kWait};
    op.other = ev.stream;
    op.upto = ev.at;
    merge(streams[s].clock, ev.clock);
    enqueue(s, op, false);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = (cudaEvent_t) new Event, cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete (Event *)e, cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    LOCK;
    Event &ev = *(Event *)e;
    merge(streams[s].clock, host);
    ev.stream = s;
    ev.at = streams[s].enqueued;
    ev.clock = streams[s].clock;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    LOCK;
    Event &ev = *(Event *)e;
    host_waits(ev.stream, ev.at, ev.clock);
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e)
{
    LOCK;
    Event &ev = *(Event *)e;
    if (!auto_progress && streams[ev.stream].done < ev.at)
        return cudaErrorNotReady;
    return cudaEventSynchronize(e);
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, enum cudaMemcpyKind, cudaStream_t s)
{
    LOCK;
    if (fails("cudaMemcpyAsync"))
        return cudaErrorInvalidValue;
    Op op{Op::kWork};
    if (is_pinned(src)) { // (pageable memory is staged before the call returns)
        op.kind = Op::kCopy;
        op.dst = dst, op.src = src, op.n = n;
        op.hash = hash_of(src, n);
    }
    enqueue(s, op, true);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *, size_t, const void *, size_t, size_t, size_t, enum cudaMemcpyKind, cudaStream_t s)
{
    return launch("cudaMemcpy2DAsync", s);
}
cudaError_t cudaMemcpy(void *dst, const void *src, size_t n, enum cudaMemcpyKind)
{
    LOCK;
    device_calls++;
    memcpy(dst, src, n);
    return cudaStreamSynchronize(nullptr);
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t s) { return launch("cudaMemsetAsync", s); }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode)
{
    LOCK;
    streams[s].capturing = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *gr)
{
    LOCK;
    streams[s].capturing = false;
    *gr = (cudaGraph_t)1;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long)
{
    return *e = (cudaGraphExec_t)1, cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { return launch("cudaGraphLaunch", s); }
} // extern "C"

namespace sgl {
cudaError_t launch_world(const SceneDev &, bool, float4 *, cudaStream_t st) { return launch("launch_world", st); }
cudaError_t launch_poses(const PoseDev *, int, uint32_t, uint32_t, cudaStream_t st) { return launch("launch_poses", st); }
cudaError_t launch_batch(const BatchDev *, int, int, cudaStream_t st, int *, Profiler *)
{
    return launch("launch_batch", st);
}
cudaError_t launch_dof(const BatchDev *, cudaStream_t st) { return launch("launch_dof", st); }
cudaError_t init_device_constants() { return cudaSuccess; }
cudaError_t check_status(unsigned *, unsigned long long *, unsigned *, bool, bool *compiled)
{
    return *compiled = false, cudaSuccess;
}
const char *prof_kernel_name(int) { return "?"; }
void prof_flush(Profiler *) {}
} // namespace sgl

// Streams of the test's own.
cudaStream_t test_stream()
{
    cudaStream_t s;
    cudaStreamCreateWithFlags(&s, 0);
    streams[s].by_test = true;
    return s;
}
