// Ray-query service (extension entry points prgpu_trace_rays / prgpu_accel_*): closest-hit and
// any-hit traversal of 32-byte rays against a converted caller BVH. One thread per ray over a
// grid sized in multiples of the SM count; rays are read as two 16-byte vector loads and
// results written as coalesced 4-byte stores.

#include <algorithm>
#include <map>
#include <memory>

#include "accel.cuh"

namespace prb {

// Persistent warps: the lanes advance their traversals one node or leaf per iteration, and lanes
// whose ray is done take the next rays from a global counter (one atomic per warp and refill).
// Incoherent rays end after very different numbers of steps; refilling keeps the lanes of a warp
// busy instead of idling until the warp's longest ray ends. A refill (ray load, reciprocal
// direction, root-box test, and the finished rays' result stores) runs once kRefillLanes lanes of
// the warp are idle, or none is busy.
// kTail (4-wide form): a query with fewer rays than the grid has lanes is spread over the warps, and once
// the queue has run dry a warp finishes its last rays with all its lanes (traverse4_finish).

template <bool kAny, bool kWide, bool kTail>
__global__ void __launch_bounds__(256, 4) k_trace_persist(const void *__restrict__ nodes,
                                                          const LeafPrim *__restrict__ prims, RootInfo root,
                                                          const float4 *__restrict__ rays, int64_t n,
                                                          int32_t *__restrict__ primOut, float *__restrict__ tOut,
                                                          float *__restrict__ b1Out, float *__restrict__ b2Out,
                                                          int *__restrict__ status,
                                                          unsigned long long *__restrict__ counter) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int stackRef[kStackSize];
    float stackT[kStackSize];
    // The 4-wide traversal keeps the bottom of its stack in shared memory.
    __shared__ int2 shortStack[kShortStack * 256];
    HybridStack<kShortStack, 256> hs;
    hs.sh = shortStack + threadIdx.x;
    TraceRay r;
    TravState s;
    s.ref = 0;
    s.sp = 0;
    s.tMax = 0.f;
    s.found = false;
    s.hit.prim = -1;
    int64_t idx = 0;
    // pending: this lane's last ray is finished and its result not yet stored.
    bool active = false, exhausted = false, pending = false, overflow = false;
    const int64_t warps = int64_t(gridDim.x) * (blockDim.x / 32);
    if (kTail && lane >= (n + warps - 1) / warps) exhausted = true;
    bool drained = false;
    auto store = [&]() {
        if (kAny) {
            primOut[idx] = s.found ? 1 : 0;
        } else if (kWide) {
            const Hit h = finish_hit<false>(prims, r, s);
            primOut[idx] = h.prim;
            if (tOut) tOut[idx] = h.t;
            if (b1Out) b1Out[idx] = h.u;
            if (b2Out) b2Out[idx] = h.v;
        } else {
            primOut[idx] = s.found ? s.hit.prim : -1;
            if (tOut) tOut[idx] = s.found ? s.hit.t : 0.f;
            if (b1Out) b1Out[idx] = s.found ? s.hit.u : 0.f;
            if (b2Out) b2Out[idx] = s.found ? s.hit.v : 0.f;
        }
    };
    while (true) {
        const bool idle = !active && !exhausted;
        const unsigned need = __ballot_sync(full, idle), busy = __ballot_sync(full, active);
        if (need && (__popc(need) >= kRefillLanes || !busy)) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(counter, (unsigned long long)__popc(need));
            base = __shfl_sync(full, base, 0);
            if (idle) {
                if (pending) store();
                idx = int64_t(base) + __popc(need & ((1u << lane) - 1u));
                if (idx >= n) {
                    exhausted = true;
                    pending = false;
                } else {
                    float4 a = __ldcs(rays + 2 * idx), b = __ldcs(rays + 2 * idx + 1);
                    r = make_trace_ray(mk(a.x, a.y, a.z), mk(b.x, b.y, b.z));
                    s.tMax = a.w;
                    s.sp = 0;
                    s.found = false;
                    s.hit.prim = -1;
                    float te;
                    active = !root.empty &&
                             box_entry(r, root.box[0], root.box[1], root.box[2], root.box[3], root.box[4], root.box[5], &te) &&
                             te < s.tMax;
                    s.ref = root.ref;
                    // A ray that misses the root is done at once: a miss, stored at the next refill.
                    pending = !active;
                }
            }
            drained = kTail && root.bound <= kCoopBound && __any_sync(full, exhausted);
            continue;
        }
        if (!busy) break;
        bool done = false;
        if (kWide) {
            // The queue has run dry and few rays are left: the warp finishes them together, below.
            if (kTail && drained && coop_ready(busy, active, s.sp)) break;
            if (leaf_turn(busy, __ballot_sync(full, active && s.ref < 0))) {
                if (active && s.ref < 0) done = traverse4_leaf<kAny, false, false, true>(prims, r, s, hs);
            } else if (active && s.ref >= 0) {
                done = traverse4_node<kAny, true>(static_cast<const QNode *>(nodes), r, s, hs, &overflow);
            }
        } else if (active) {
            done = traverse_step<kAny, false>(static_cast<const WNode *>(nodes), prims, r, s, stackRef, stackT, &overflow);
        }
        if (done) {
            active = false;
            pending = true;
        }
    }
    if (kTail) {
        if (__any_sync(full, active)) {
            const float tMax = active ? __ldcs(&rays[2 * idx].w) : 0.f;
            overflow |= traverse4_finish<kAny, false, false, false>(static_cast<const QNode *>(nodes), prims, nullptr,
                                                                    root.bound, root.ref, r, s, active, hs, tMax);
        }
        if (active || pending) store();
    }
    if (overflow) atomicOr(status, 1);
}

// Resident blocks per SM of a kernel (asked once): the persistent grid is exactly one full wave.
template <bool kAny, bool kWide, bool kTail> int resident_blocks(int block) {
    static const int n = [block] {
        int k = 0;
        PRB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, k_trace_persist<kAny, kWide, kTail>, block, 0));
        return std::max(1, k);
    }();
    return n;
}

// A query: device pointers, its status word, and a ray counter that no query that may run at the same
// time uses (RayCounters).
struct TraceArgs {
    const prgpu::Ray *rays;
    int64_t n;
    int32_t *prim;
    float *t, *b1, *b2;
    int *status;
    unsigned long long *counter;
    cudaStream_t stream;
    int smCount;
};

// raysPerBlock: one ray a lane, or (tail form) down to one a warp.
template <bool kAny, bool kWide, bool kTail> void launch_one(const DeviceAccel &acc, const TraceArgs &q) {
    const int block = 256, raysPerBlock = kTail ? block / 32 : block;
    const int64_t needed = (q.n + raysPerBlock - 1) / raysPerBlock;
    const int grid = int(std::min<int64_t>(needed, int64_t(q.smCount) * resident_blocks<kAny, kWide, kTail>(block)));
    PRB_CUDA(cudaMemsetAsync(q.counter, 0, sizeof(*q.counter), q.stream));
    k_trace_persist<kAny, kWide, kTail><<<grid, block, 0, q.stream>>>(
        kWide ? acc.qnodes.ptr : acc.nodes.ptr, acc.prims.as<LeafPrim>(), acc.root,
        reinterpret_cast<const float4 *>(q.rays), q.n, q.prim, kAny ? nullptr : q.t, kAny ? nullptr : q.b1,
        kAny ? nullptr : q.b2, q.status, q.counter);
    count_launch();
    PRB_CUDA(cudaGetLastError());
}

// Closest hits: up to this many rays the launch's tail, 35 to 60 us with one lane a ray to the end, costs
// more than the registers that the call of traverse4_finish takes from the loop (5 %). us, one lane / tail
// form: 1M-triangle soup, 4,096 rays 129 / 84, 262,144 254 / 205, 1.5M 557 / 504, 2.1M 665 / 650, 4.2M
// 1142 / 1155, 16.8M 3987 / 4207; 100,003 triangles, 4.2M rays 1012 / 991, 8.4M 1812 / 1868; 4,096
// triangles, 2.1M rays 441 / 432, 4.2M 775 / 787.
// Any hits take the tail form at every size, as its loop spills nothing: 4,096 rays 111 / 57, 1.5M 420 / 354,
// 4.2M 857 / 777, 16.8M 2791 / 2716; 4,096 triangles, 16.8M rays 1977 / 1949.
constexpr int64_t kTailRays = 3 << 20;

// wide: the 4-wide tree, each ray's hit a function of the ray and the tree alone; otherwise the binary
// tree in the reference's visit order (bvh.cpp:184-190). The two visit leaves in different orders, which
// shows among hits at exactly equal distances, or closer together than the rounding of a box's entry.
void launch_trace(const DeviceAccel &acc, const TraceArgs &q, bool anyHit, bool wide) {
    if (q.n <= 0) return;
    if (!wide) {
        if (anyHit) launch_one<true, false, false>(acc, q);
        else launch_one<false, false, false>(acc, q);
    } else if (anyHit) {
        launch_one<true, true, true>(acc, q);
    } else if (q.n <= kTailRays) {
        launch_one<false, true, true>(acc, q);
    } else {
        launch_one<false, true, false>(acc, q);
    }
}

// The ray counters of a handle. A query resets its counter and draws its rays from it, so queries that
// may overlap on the device need one each, while those of one stream run one after another and share
// one: a counter per stream, by the stream's id, which is never used again (its address is). What is
// captured runs later, on any stream and any number of times: a counter of its own for each such query.
class RayCounters {
  public:
    // The first `count` counters lie in the caller's memory at p, kStride bytes each.
    static constexpr size_t kStride = 32;
    void init(void *p, size_t count) {
        next_ = static_cast<char *>(p);
        left_ = count;
    }
    unsigned long long *of(cudaStream_t stream) {
        cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
        PRB_CUDA(cudaStreamIsCapturing(stream, &capturing));
        if (capturing != cudaStreamCaptureStatusNone) return take();
        unsigned long long id = 0;
        PRB_CUDA(cudaStreamGetId(stream, &id));
        unsigned long long *&c = known_[id];
        if (!c) c = take();
        return c;
    }
    void release() {
        for (DevBuf &b : more_) b.release();
        more_.clear();
        known_.clear();
    }

  private:
    unsigned long long *take() {
        if (!left_) grow();
        auto *c = reinterpret_cast<unsigned long long *>(next_);
        next_ += kStride;
        --left_;
        return c;
    }
    void grow() {
        const size_t count = 4096;
        more_.emplace_back();
        // Also while this or another thread captures: an allocation is no part of what is captured.
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        PRB_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
        const cudaError_t e = cudaMalloc(&more_.back().ptr, count * kStride);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) more_.pop_back();
        check_cuda(e, "cudaMalloc of ray counters");
        init(more_.back().ptr, count);
    }
    std::map<unsigned long long, unsigned long long *> known_;
    std::vector<DevBuf> more_;
    char *next_ = nullptr;
    size_t left_ = 0;
};

} // namespace prb

using namespace prb;

struct prgpu_accel_t {
    DeviceAccel acc;
    int device = -1;
    DevBuf status;  // two status words (queries on device buffers, on host buffers), then ray counters
    DevBuf rays, prim, t, b1, b2;  // staging for the host-buffer path
    std::mutex mutex;              // the counters, and a counter's reset with the launch that draws from it
    RayCounters counters;
    std::atomic<int> hostStatus{0};  // what host-buffer queries reported, for prgpu_accel_status

    void trace(TraceArgs q, bool anyHit, bool wide) {
        std::lock_guard<std::mutex> lock(mutex);
        q.counter = counters.of(q.stream);
        launch_trace(acc, q, anyHit, wide);
    }
    void release() {
        acc.release();
        counters.release();
        for (DevBuf *b : {&status, &rays, &prim, &t, &b1, &b2}) b->release();
    }
};

namespace {

bool make_accel(int deviceIndex, const prgpu::BVHNode *nodes, int32_t nodeCount, const int32_t *primOrder,
                const prgpu::Float3 *triVerts, int32_t primCount, prgpu_accel_t *a, std::string *err) {
    if (primCount > 0 && !triVerts) {
        *err = "null triangle array";
        return false;
    }
    HostAccel h;
    if (!convert_bvh(nodes, nodeCount, primOrder, primCount, TriangleSoupSource{triVerts}, &h, err)) return false;
    DeviceState &ds = device_state(deviceIndex);
    a->device = ds.device;
    a->acc.upload(h, ds.stream);
    const size_t counters = 255;
    a->status.ensure((1 + counters) * RayCounters::kStride);
    a->counters.init(a->status.as<char>() + RayCounters::kStride, counters);
    PRB_CUDA(cudaMemsetAsync(a->status.ptr, 0, 2 * sizeof(int), ds.stream));
    PRB_CUDA(cudaStreamSynchronize(ds.stream));
    return true;
}

// Host-buffer query: rays are copied in chunks on the copy stream while the previous chunk is
// traced on the compute stream; results are copied back per chunk. The call is bound by the
// host-to-device copy (32 B per ray in, 4-8 B out); chunks of 2^20 rays (32 MiB) keep the copy
// engine busy while a chunk's trace and result copy (well under its copy time) overlap the next
// chunk's copy, and keep the unoverlapped first copy and last trace of a call short.
bool trace_host(prgpu_accel_t *a, const prgpu::Ray *rays, int64_t n, int anyHit, int32_t *primOut, float *tOut,
                float *b1Out, float *b2Out, bool wide, std::string *err) {
    DeviceState &ds = device_state(a->device);
    const int64_t chunk = int64_t(1) << 20;
    int64_t cap = std::min<int64_t>(n, 2 * chunk);
    a->rays.ensure(size_t(std::max<int64_t>(cap, 1)) * sizeof(prgpu::Ray));
    a->prim.ensure(size_t(std::max<int64_t>(cap, 1)) * sizeof(int32_t));
    if (tOut) a->t.ensure(size_t(std::max<int64_t>(cap, 1)) * sizeof(float));
    if (b1Out) a->b1.ensure(size_t(std::max<int64_t>(cap, 1)) * sizeof(float));
    if (b2Out) a->b2.ensure(size_t(std::max<int64_t>(cap, 1)) * sizeof(float));
    int *dStatus = a->status.as<int>() + 1;
    PRB_CUDA(cudaMemsetAsync(dStatus, 0, sizeof(int), ds.stream));
    cudaEvent_t copied[2], traced[2];
    for (int k = 0; k < 2; ++k) {
        PRB_CUDA(cudaEventCreateWithFlags(&copied[k], cudaEventDisableTiming));
        PRB_CUDA(cudaEventCreateWithFlags(&traced[k], cudaEventDisableTiming));
    }
    int64_t nChunks = (n + chunk - 1) / chunk;
    for (int64_t c = 0; c < nChunks; ++c) {
        int slot = int(c & 1);
        int64_t off = c * chunk, cnt = std::min(chunk, n - off);
        int64_t base = int64_t(slot) * chunk;
        // The slot's previous results must be back on the host before it is overwritten.
        if (c >= 2) PRB_CUDA(cudaStreamWaitEvent(ds.copy, traced[slot], 0));
        PRB_CUDA(cudaMemcpyAsync(a->rays.as<prgpu::Ray>() + base, rays + off, size_t(cnt) * sizeof(prgpu::Ray),
                                 cudaMemcpyHostToDevice, ds.copy));
        PRB_CUDA(cudaEventRecord(copied[slot], ds.copy));
        PRB_CUDA(cudaStreamWaitEvent(ds.stream, copied[slot], 0));
        a->trace({a->rays.as<prgpu::Ray>() + base, cnt, a->prim.as<int32_t>() + base,
                  tOut ? a->t.as<float>() + base : nullptr, b1Out ? a->b1.as<float>() + base : nullptr,
                  b2Out ? a->b2.as<float>() + base : nullptr, dStatus, nullptr, ds.stream, ds.prop.multiProcessorCount},
                 anyHit != 0, wide);
        PRB_CUDA(cudaMemcpyAsync(primOut + off, a->prim.as<int32_t>() + base, size_t(cnt) * sizeof(int32_t),
                                 cudaMemcpyDeviceToHost, ds.stream));
        if (tOut)
            PRB_CUDA(cudaMemcpyAsync(tOut + off, a->t.as<float>() + base, size_t(cnt) * sizeof(float),
                                     cudaMemcpyDeviceToHost, ds.stream));
        if (b1Out)
            PRB_CUDA(cudaMemcpyAsync(b1Out + off, a->b1.as<float>() + base, size_t(cnt) * sizeof(float),
                                     cudaMemcpyDeviceToHost, ds.stream));
        if (b2Out)
            PRB_CUDA(cudaMemcpyAsync(b2Out + off, a->b2.as<float>() + base, size_t(cnt) * sizeof(float),
                                     cudaMemcpyDeviceToHost, ds.stream));
        PRB_CUDA(cudaEventRecord(traced[slot], ds.stream));
    }
    int status = 0;
    PRB_CUDA(cudaMemcpyAsync(&status, dStatus, sizeof(int), cudaMemcpyDeviceToHost, ds.stream));
    PRB_CUDA(cudaStreamSynchronize(ds.stream));
    PRB_CUDA(cudaStreamSynchronize(ds.copy));
    for (int k = 0; k < 2; ++k) {
        cudaEventDestroy(copied[k]);
        cudaEventDestroy(traced[k]);
    }
    a->hostStatus |= status;
    if (status & 1) {
        *err = "BVH deeper than the traversal stack (64 entries)";
        return false;
    }
    return true;
}

} // namespace

PRGPU_API int prgpu_trace_rays(int deviceIndex, const prgpu::BVHNode *nodes, int32_t nodeCount, const int32_t *primOrder,
                               const prgpu::Float3 *triVerts, int32_t primCount, const prgpu::Ray *rays, int64_t rayCount,
                               int32_t anyHit, int32_t *primOut, float *tOut, float *b1Out, float *b2Out, char *err,
                               int errLen) {
    std::lock_guard<std::mutex> lock(gApiMutex);
    try {
        if (rayCount < 0 || (rayCount > 0 && (!rays || !primOut))) {
            set_err(err, errLen, "bad ray arguments");
            return 1;
        }
        prgpu_accel_t a;
        std::string e;
        bool ok = make_accel(deviceIndex, nodes, nodeCount, primOrder, triVerts, primCount, &a, &e) &&
                  trace_host(&a, rays, rayCount, anyHit, primOut, tOut, b1Out, b2Out, false, &e);
        a.release();
        if (!ok) {
            set_err(err, errLen, e);
            return 1;
        }
        return 0;
    } catch (const CudaError &e) {
        set_err(err, errLen, e.msg);
        return 1;
    } catch (const std::exception &e) {
        set_err(err, errLen, e.what());
        return 1;
    }
}

PRGPU_API int prgpu_accel_create(int deviceIndex, const prgpu::BVHNode *nodes, int32_t nodeCount, const int32_t *primOrder,
                                 const prgpu::Float3 *triVerts, int32_t primCount, prgpu_accel *out, char *err,
                                 int errLen) {
    std::lock_guard<std::mutex> lock(gApiMutex);
    if (!out) {
        set_err(err, errLen, "null output handle");
        return 1;
    }
    *out = nullptr;
    try {
        auto a = std::make_unique<prgpu_accel_t>();
        std::string e;
        if (!make_accel(deviceIndex, nodes, nodeCount, primOrder, triVerts, primCount, a.get(), &e)) {
            set_err(err, errLen, e);
            return 1;
        }
        *out = a.release();
        return 0;
    } catch (const CudaError &e) {
        set_err(err, errLen, e.msg);
        return 1;
    } catch (const std::exception &e) {
        set_err(err, errLen, e.what());
        return 1;
    }
}

PRGPU_API int prgpu_accel_trace(prgpu_accel accel, const prgpu::Ray *deviceRays, int64_t rayCount, int32_t anyHit,
                                int32_t *devicePrimOut, float *deviceTOut, void *stream, char *err, int errLen) {
    if (!accel || rayCount < 0 || (rayCount > 0 && (!deviceRays || !devicePrimOut))) {
        set_err(err, errLen, "bad arguments");
        return 1;
    }
    try {
        DeviceState &ds = device_state(accel->device);
        accel->trace({deviceRays, rayCount, devicePrimOut, deviceTOut, nullptr, nullptr, accel->status.as<int>(), nullptr,
                      static_cast<cudaStream_t>(stream), ds.prop.multiProcessorCount},
                     anyHit != 0, true);
        return 0;
    } catch (const CudaError &e) {
        set_err(err, errLen, e.msg);
        return 1;
    } catch (const std::exception &e) {
        set_err(err, errLen, e.what());
        return 1;
    }
}

// Host-buffer query against a device-resident BVH (the end-to-end path: rays in and results out
// cross the host link inside the call).
PRGPU_API int prgpu_accel_trace_host(prgpu_accel accel, const prgpu::Ray *rays, int64_t rayCount, int32_t anyHit,
                                     int32_t *primOut, float *tOut, char *err, int errLen) {
    std::lock_guard<std::mutex> lock(gApiMutex);
    if (!accel || rayCount < 0 || (rayCount > 0 && (!rays || !primOut))) {
        set_err(err, errLen, "bad arguments");
        return 1;
    }
    try {
        std::string e;
        if (!trace_host(accel, rays, rayCount, anyHit, primOut, tOut, nullptr, nullptr, true, &e)) {
            set_err(err, errLen, e);
            return 1;
        }
        return 0;
    } catch (const CudaError &e) {
        set_err(err, errLen, e.msg);
        return 1;
    } catch (const std::exception &e) {
        set_err(err, errLen, e.what());
        return 1;
    }
}

// Reads back and clears the accel's status (bit 0: a traversal stack overflowed), once all queries queued
// so far, on whatever stream, have run.
PRGPU_API int prgpu_accel_status(prgpu_accel accel) {
    if (!accel) return -1;
    try {
        device_state(accel->device);
        int s = 0;
        PRB_CUDA(cudaDeviceSynchronize());
        PRB_CUDA(cudaMemcpy(&s, accel->status.ptr, sizeof(int), cudaMemcpyDeviceToHost));
        if (s) PRB_CUDA(cudaMemset(accel->status.ptr, 0, sizeof(int)));
        return s | accel->hostStatus.exchange(0);
    } catch (const CudaError &) {
        return -1;
    }
}

PRGPU_API int64_t prgpu_accel_bytes(prgpu_accel accel) { return accel ? accel->acc.bytes : 0; }

PRGPU_API void prgpu_accel_destroy(prgpu_accel accel) {
    if (!accel) return;
    std::lock_guard<std::mutex> lock(gApiMutex);
    if (accel->device >= 0) cudaSetDevice(accel->device);
    accel->release();
    delete accel;
}
