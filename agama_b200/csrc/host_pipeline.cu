// Chunked host-array batches: copies of one chunk overlap the kernels of the others.
#include "host_pipeline.h"
#include "runtime.h"
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdint>
#include <cstring>
#include <exception>
#include <map>
#include <memory>
#include <mutex>
#include <thread>

namespace agb {

namespace {

constexpr int NUM_STREAMS = 3;
constexpr long MIN_CHUNK = 65536;
constexpr long MAX_CHUNK = 1L << 20;
constexpr size_t ALIGN = 256;

/// staging of pageable inputs: pieces of a megabyte through a ring of page-locked memory
constexpr size_t PIECE = 1 << 20;
constexpr int RING = 16, STAGING_THREADS = 4;
/// smaller inputs are copied as they are: starting the threads and handing over the pieces costs ~0.4 ms,
/// which the faster copies earn back from here on (copied / staged at 4, 16, 24, 28, 48 MB: potentials
/// 0.36 / 0.85, 1.00 / 1.15, 1.41 / 1.33, 1.65 / 1.52, 4.0 / 2.1 ms; actions 0.53 / 0.96, 1.30 / 1.64,
/// 1.81 / 1.70, 2.12 / 1.88, 3.7 / 2.6 ms)
constexpr size_t MIN_STAGED = 28 * PIECE;
constexpr size_t MAX_IDLE_RINGS = 4;            // rings kept by stream sets that are not in use

/// a set of non-blocking streams of one device, with its staging ring (allocated when first needed),
/// reused across calls (one caller at a time)
struct StreamSet {
    int device;
    cudaStream_t s[NUM_STREAMS];
    char* ring = nullptr;
    cudaEvent_t copied[RING] = {};              // the copy out of each place of the ring
};

std::mutex g_mutex;
std::vector<StreamSet*> g_idle;
std::map<int, cudaMemPool_t> g_pools;

StreamSet* acquireStreams(int device)
{
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        for(size_t i = 0; i < g_idle.size(); i++)
            if(g_idle[i]->device == device) {
                StreamSet* s = g_idle[i];
                g_idle.erase(g_idle.begin() + i);
                return s;
            }
    }
    StreamSet* s = new StreamSet;
    s->device = device;
    for(int k = 0; k < NUM_STREAMS; k++)
        AGB_CUDA(cudaStreamCreateWithFlags(&s->s[k], cudaStreamNonBlocking));
    return s;
}

/// false if there is no page-locked memory left for a ring (the inputs are then copied as they are)
bool allocateRing(StreamSet* s)
{
    if(s->ring) return true;
    for(int k = 0; k < RING; k++)
        if(!s->copied[k]) AGB_CUDA(cudaEventCreateWithFlags(&s->copied[k], cudaEventDisableTiming));
    if(cudaHostAlloc(reinterpret_cast<void**>(&s->ring), RING * PIECE, cudaHostAllocPortable) == cudaSuccess) return true;
    cudaGetLastError();
    s->ring = nullptr;
    return false;
}

void releaseStreams(StreamSet* s)
{
    char* surplus = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        size_t rings = 0;
        for(const StreamSet* i : g_idle) rings += i->ring != nullptr;
        if(s->ring && rings >= MAX_IDLE_RINGS) std::swap(surplus, s->ring);
        g_idle.push_back(s);
    }
    if(surplus) cudaFreeHost(surplus);
}

/// one piece of an input on its way to the device
struct Piece { const char* src; char* dst; size_t bytes; };

/** The pieces of a call's pageable inputs, in order, copied into the ring by a few threads while the
    caller issues the copies to the device: a copy from pageable memory runs at the speed of one
    thread's copy inside the driver and holds the caller until it is done (2.4 ms for the 34 MB of 7e5
    phase-space points, longer than their kernels), while from page-locked memory it is asynchronous.
    Actions of 7e5 halo points of pageable memory: 3528 -> 2393 us. */
class Stager {
public:
    Stager(StreamSet* set, std::vector<Piece> list) : set_(set), pieces_(std::move(list)),
        ready_(new std::atomic<int>[pieces_.size()])
    {
        for(size_t p = 0; p < pieces_.size(); p++) ready_[p] = 0;
        const size_t cores = std::max(1u, std::thread::hardware_concurrency());
        const size_t count = std::min({ static_cast<size_t>(STAGING_THREADS), cores, pieces_.size() });
        threads_.reserve(count);
        try {
            for(size_t t = 0; t < count; t++) threads_.emplace_back([this] { work(); });
        } catch(const std::exception&) {}       // no thread or no memory for one more: the ones that run do the work
    }
    bool running() const { return !threads_.empty(); }
    ~Stager()
    {
        stop_ = true;
        for(std::thread& t : threads_) t.join();
    }
    Stager(const Stager&) = delete;
    Stager& operator=(const Stager&) = delete;

    /// copy the next piece to the device on the stream, as soon as it is in the ring
    void issue(cudaStream_t stream)
    {
        const size_t p = issued_;
        for(int k = 0; !ready_[p]; k++) {
            if(failed_) throw std::runtime_error("CUDA error: staging of a host array failed");
            pause(k);
        }
        AGB_CUDA(cudaMemcpyAsync(pieces_[p].dst, set_->ring + p % RING * PIECE, pieces_[p].bytes, cudaMemcpyHostToDevice,
            stream));
        AGB_CUDA(cudaEventRecord(set_->copied[p % RING], stream));
        issued_ = p + 1;
    }

private:
    /// waits are short (a piece takes 0.1 ms) unless the caller is held by a copy of results
    static void pause(int k)
    {
        if(k < 1000) std::this_thread::yield();
        else std::this_thread::sleep_for(std::chrono::microseconds(50));
    }

    void work()
    {
        if(cudaSetDevice(set_->device) != cudaSuccess) { failed_ = true; return; }
        while(!stop_) {
            const size_t p = next_++;
            if(p >= pieces_.size()) return;
            if(p >= RING) {     // the place's previous piece has to be on the device
                for(int k = 0; issued_ <= p - RING; k++) {
                    if(stop_) return;
                    pause(k);
                }
                if(cudaEventSynchronize(set_->copied[p % RING]) != cudaSuccess) { failed_ = true; return; }
            }
            memcpy(set_->ring + p % RING * PIECE, pieces_[p].src, pieces_[p].bytes);
            ready_[p] = 1;
        }
    }

    StreamSet* set_;
    std::vector<Piece> pieces_;
    std::unique_ptr<std::atomic<int>[]> ready_;
    std::atomic<size_t> next_{ 0 }, issued_{ 0 };
    std::atomic<bool> stop_{ false }, failed_{ false };
    std::vector<std::thread> threads_;
};

/// memory that the driver would have to copy itself (neither page-locked nor of a device)
bool isPageable(const void* p)
{
    cudaPointerAttributes a;
    if(cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type == cudaMemoryTypeUnregistered;
}

/// the engine's own pool on a device (not the device's default pool, whose settings belong to
/// the application): memory freed back to it stays reserved for the next call
cudaMemPool_t poolFor(int device)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    auto it = g_pools.find(device);
    if(it != g_pools.end()) return it->second;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool;
    AGB_CUDA(cudaMemPoolCreate(&pool, &props));
    uint64_t threshold = UINT64_MAX;
    AGB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &threshold));
    // a block freed on one stream is not handed to an allocation on another: such reuse makes
    // the allocating stream wait for the freeing one, which serialised the chunks of a host-buffer
    // call (each chunk's scratch on its own stream) instead of overlapping their kernels
    int off = 0;
    AGB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolReuseFollowEventDependencies, &off));
    AGB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowOpportunistic, &off));
    AGB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &off));
    g_pools[device] = pool;
    return pool;
}

size_t roundUp(size_t x) { return (x + ALIGN - 1) / ALIGN * ALIGN; }

/// scratch and streams of one call; the destructor waits for the streams and returns both,
/// also when the call is left by an exception
struct Call {
    StreamSet* streams = nullptr;
    char* scratch[NUM_STREAMS] = {};
    ~Call() {
        if(!streams) return;
        for(int k = 0; k < NUM_STREAMS; k++) {
            if(scratch[k]) cudaFreeAsync(scratch[k], streams->s[k]);
            cudaStreamSynchronize(streams->s[k]);
        }
        releaseStreams(streams);
    }
};

}  // namespace

void* scratchAlloc(size_t bytes, cudaStream_t stream)
{
    int device;
    AGB_CUDA(cudaGetDevice(&device));
    void* p = nullptr;
    AGB_CUDA(cudaMallocFromPoolAsync(&p, std::max<size_t>(bytes, ALIGN), poolFor(device), stream));
    return p;
}

void scratchFree(void* ptr, cudaStream_t stream)
{
    if(ptr) cudaFreeAsync(ptr, stream);
}

void runChunked(long n, const std::vector<HostIn>& ins, const std::vector<HostOut>& outs,
    const ChunkLaunch& launch, long chunk)
{
    if(n <= 0) return;
    // chunk boundaries (a given chunk size, or the default below)
    std::vector<long> bounds{ 0 };
    if(chunk > 0) {
        for(long f = chunk; f < n; f += chunk) bounds.push_back(f);
    } else if(n >= 8 * MIN_CHUNK) {
        // a short first chunk (its copy in is exposed) and chunks growing so that each copy in
        // ends before the kernels of the previous chunk do; a short last chunk (its copy out is
        // exposed): fractions 0.05, 0.20, 0.35, 0.30, 0.10 of n
        const double frac[4] = { 0.05, 0.25, 0.60, 0.90 };
        for(double f : frac) bounds.push_back(static_cast<long>(f * n));
    } else {        // small batches: four chunks of at least MIN_CHUNK items
        const long c = std::min(MAX_CHUNK, std::max(MIN_CHUNK, (n + 3) / 4));
        for(long f = c; f < n; f += c) bounds.push_back(f);
    }
    bounds.push_back(n);
    for(size_t k = 0; k + 1 < bounds.size(); k++)      // no chunk above the scratch bound
        if(bounds[k + 1] - bounds[k] > MAX_CHUNK) { bounds.insert(bounds.begin() + k + 1, bounds[k] + MAX_CHUNK); }
    const long numChunks = static_cast<long>(bounds.size()) - 1;
    chunk = 0;
    for(long c = 0; c < numChunks; c++) chunk = std::max(chunk, bounds[c + 1] - bounds[c]);
    const int slots = static_cast<int>(std::min<long>(NUM_STREAMS, numChunks));
    int device;
    AGB_CUDA(cudaGetDevice(&device));
    cudaMemPool_t pool = poolFor(device);

    // per-slot scratch: every used array of one chunk, each 256-byte aligned
    std::vector<size_t> inOff(ins.size()), outOff(outs.size());
    size_t bytes = 0;
    for(size_t a = 0; a < ins.size(); a++) { inOff[a] = bytes; if(ins[a].host) bytes += roundUp(ins[a].itemBytes * chunk); }
    for(size_t a = 0; a < outs.size(); a++) { outOff[a] = bytes; if(outs[a].host) bytes += roundUp(outs[a].itemBytes * chunk); }

    Call call;
    call.streams = acquireStreams(device);
    for(int k = 0; k < slots; k++)
        AGB_CUDA(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&call.scratch[k]), std::max<size_t>(bytes, ALIGN),
            pool, call.streams->s[k]));

    // large pageable inputs go through the staging ring, piece by piece in the order of the chunks
    std::vector<bool> staged(ins.size());
    size_t stagedBytes = 0;
    for(size_t a = 0; a < ins.size(); a++)
        if(ins[a].host && ins[a].itemBytes * n >= MIN_STAGED && isPageable(ins[a].host)) {
            staged[a] = true;
            stagedBytes += ins[a].itemBytes * n;
        }
    std::unique_ptr<Stager> stager;
    std::vector<std::vector<int>> pieceCount(numChunks, std::vector<int>(ins.size(), 0));
    if(stagedBytes && allocateRing(call.streams)) {
        std::vector<Piece> pieces;
        for(long c = 0; c < numChunks; c++)
            for(size_t a = 0; a < ins.size(); a++) {
                if(!staged[a]) continue;
                const char* src = static_cast<const char*>(ins[a].host) + bounds[c] * ins[a].itemBytes;
                const size_t size = (bounds[c + 1] - bounds[c]) * ins[a].itemBytes;
                for(size_t f = 0; f < size; f += PIECE, pieceCount[c][a]++)
                    pieces.push_back(Piece{ src + f, call.scratch[c % slots] + inOff[a] + f, std::min(PIECE, size - f) });
            }
        stager.reset(new Stager(call.streams, std::move(pieces)));
        if(!stager->running()) stager.reset();
    }

    std::vector<void*> dIn(ins.size()), dOut(outs.size());
    auto copyOut = [&](long c) {
        const int k = static_cast<int>(c % slots);
        const long first = bounds[c], count = bounds[c + 1] - bounds[c];
        for(size_t a = 0; a < outs.size(); a++)
            if(outs[a].host)
                AGB_CUDA(cudaMemcpyAsync(static_cast<char*>(outs[a].host) + first * outs[a].itemBytes,
                    call.scratch[k] + outOff[a], count * outs[a].itemBytes, cudaMemcpyDefault, call.streams->s[k]));
    };
    // software pipeline: chunk c is copied in and launched before the copy-out of chunk c-1 is
    // issued, so that a copy-out into pageable memory (which returns only when it is done)
    // never holds back the next launch.  A slot's scratch is reused NUM_STREAMS chunks later on
    // the same stream, after its copy-out.
    for(long c = 0; c < numChunks; c++) {
        const int k = static_cast<int>(c % slots);
        const long first = bounds[c], count = bounds[c + 1] - bounds[c];
        cudaStream_t s = call.streams->s[k];
        for(size_t a = 0; a < ins.size(); a++) {
            dIn[a] = ins[a].host ? call.scratch[k] + inOff[a] : nullptr;
            if(stager && staged[a])
                for(int p = 0; p < pieceCount[c][a]; p++) stager->issue(s);
            else if(ins[a].host)
                AGB_CUDA(cudaMemcpyAsync(dIn[a], static_cast<const char*>(ins[a].host) + first * ins[a].itemBytes,
                    count * ins[a].itemBytes, cudaMemcpyDefault, s));
        }
        for(size_t a = 0; a < outs.size(); a++)
            dOut[a] = outs[a].host ? call.scratch[k] + outOff[a] : nullptr;
        launch(first, count, dIn.data(), dOut.data(), s);
        if(c > 0) copyOut(c - 1);
    }
    copyOut(numChunks - 1);
    for(int k = 0; k < slots; k++) {
        AGB_CUDA(cudaFreeAsync(call.scratch[k], call.streams->s[k]));
        call.scratch[k] = nullptr;
    }
    for(int k = 0; k < slots; k++)
        AGB_CUDA(cudaStreamSynchronize(call.streams->s[k]));
}

}  // namespace agb
