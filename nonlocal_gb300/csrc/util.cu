// Prefix sums and small helpers shared by the pattern, neighbour and solver
// stages.
#include "common.cuh"

#include <mutex>

namespace nlgpu {

std::atomic<int64_t> g_launches{0};
thread_local int64_t* t_capture_sink = nullptr;
thread_local std::shared_ptr<Arena> t_arena;

namespace {

// What is kept idle: an arena BLOCK_MAX a block and IDLE_MAX in all, the pool of a
// device POOL_MAX, all arenas and the pool of a device together DEVICE_MAX (1.4 % of its
// memory); anything above is freed at once, as it would be without them.
// (A problem whose matrices exceed BLOCK_MAX runs for tens of milliseconds, beside
// which its few large frees, 1 to 5 ms each, matter little; the small ones matter.)
constexpr size_t BLOCK_MAX = size_t(256) << 20;
constexpr size_t IDLE_MAX = size_t(1) << 30;
constexpr size_t POOL_MAX = size_t(1) << 30;
constexpr size_t DEVICE_MAX = size_t(4) << 30;

// idle blocks by size
struct IdleBlocks {
    std::mutex mutex;
    std::multimap<size_t, void*> blocks;
    size_t bytes = 0;
    std::atomic<size_t>* device_bytes = nullptr;   // idle on the device in all
    // the smallest block that holds `need` without wasting more than an eighth of
    // it (64 KB for small requests)
    void* get(size_t need, size_t* capacity) {
        std::lock_guard<std::mutex> lock{mutex};
        const auto it = blocks.lower_bound(need);
        if (it == blocks.end() || it->first > need + std::max<size_t>(need / 8, 64 << 10)) return nullptr;
        void* p = it->second;
        *capacity = it->first;
        bytes -= it->first;
        *device_bytes -= it->first;
        blocks.erase(it);
        return p;
    }
    bool put(void* p, size_t capacity, size_t limit) {
        std::lock_guard<std::mutex> lock{mutex};
        if (capacity > BLOCK_MAX || bytes + capacity > limit) return false;
        if ((*device_bytes += capacity) > DEVICE_MAX) {
            *device_bytes -= capacity;
            return false;
        }
        try {
            blocks.emplace(capacity, p);
        } catch (...) {
            *device_bytes -= capacity;
            throw;
        }
        bytes += capacity;
        return true;
    }
    // cudaFree waits for the work that may still use a block
    void give_back() {
        std::lock_guard<std::mutex> lock{mutex};
        for (const auto& b : blocks) cudaFree(b.second);
        blocks.clear();
        *device_bytes -= bytes;
        bytes = 0;
    }
};

}  // namespace

struct Arena::Blocks : IdleBlocks {};

namespace {

// the pools of the devices and every live arena; never destroyed (the driver may be
// gone when static objects end)
struct Memory {
    std::mutex mutex;
    struct Device {
        std::atomic<size_t> idle{0};
        IdleBlocks pool;
        Device() { pool.device_bytes = &idle; }
    };
    std::map<int, Device> devices;
    std::map<IdleBlocks*, int> arenas;   // with their devices
    IdleBlocks& pool(int device) {
        std::lock_guard<std::mutex> lock{mutex};
        return devices[device].pool;
    }
    void give_back(int device) {
        std::lock_guard<std::mutex> lock{mutex};
        devices[device].pool.give_back();
        for (const auto& [blocks, d] : arenas)
            if (d == device) blocks->give_back();
    }
};
Memory& memory() {
    static Memory* m = new Memory;
    return *m;
}

int current_device() {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess) {
        (void)cudaGetLastError();
        d = 0;
    }
    return d;
}

}  // namespace

Arena::Arena() : blocks{std::make_unique<Blocks>()}, device{current_device()} {
    Memory& m = memory();
    std::lock_guard<std::mutex> lock{m.mutex};
    blocks->device_bytes = &m.devices[device].idle;
    m.arenas.emplace(blocks.get(), device);
}

Arena::~Arena() {
    Memory& m = memory();
    {
        std::lock_guard<std::mutex> lock{m.mutex};
        m.arenas.erase(blocks.get());
    }
    IdleBlocks& pool = m.pool(device);
    *blocks->device_bytes -= blocks->bytes;
    for (const auto& [size, p] : blocks->blocks) {
        bool kept = false;
        try {
            kept = pool.put(p, size, POOL_MAX);
        } catch (...) {
        }
        if (!kept) cudaFree(p);
    }
}

void release_idle_memory() { memory().give_back(current_device()); }

void* Arena::get(size_t bytes, size_t* capacity) {
    bytes = (bytes + 511) / 512 * 512;
    void* p = nullptr;
    if (current_device() != device) {   // the calling thread's device decides, as ever: not a block of this arena
        NL_CUDA(cudaMalloc(&p, bytes));
        *capacity = 0;
        return p;
    }
    if ((p = blocks->get(bytes, capacity)) || (p = memory().pool(device).get(bytes, capacity))) return p;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaErrorMemoryAllocation) {   // the idle blocks of every context go back first
        (void)cudaGetLastError();
        memory().give_back(device);
        e = cudaMalloc(&p, bytes);
    }
    NL_CUDA(e);
    *capacity = bytes;
    return p;
}

void Arena::put(void* p, size_t capacity) noexcept {
    bool kept = false;
    try {
        kept = capacity && blocks->put(p, capacity, IDLE_MAX);
    } catch (...) {
    }
    if (!kept) cudaFree(p);
}

namespace {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ i64 block_exclusive_scan(i64 v, i64* sh, i64* total) {
    // sh: SCAN_THREADS / 32 entries
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    i64 incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const i64 t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) sh[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        i64 s = lane < SCAN_THREADS / 32 ? sh[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const i64 t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        if (lane < SCAN_THREADS / 32) sh[lane] = s;
    }
    __syncthreads();
    const i64 warp_off = warp ? sh[warp - 1] : 0;
    if (total) *total = sh[SCAN_THREADS / 32 - 1];
    __syncthreads();
    return warp_off + incl - v;
}

__global__ void k_tile_sums(const i64* in, i64 n, i64* sums) {
    __shared__ i64 sh[SCAN_THREADS / 32];
    const i64 base = i64(blockIdx.x) * SCAN_TILE;
    i64 s = 0;
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const i64 i = base + i64(threadIdx.x) * SCAN_ITEMS + k;
        if (i < n) s += in[i];
    }
    i64 total;
    block_exclusive_scan(s, sh, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void k_scan_sums(i64* sums, i64 nb, i64* grand_total) {
    __shared__ i64 sh[SCAN_THREADS / 32];
    i64 carry = 0;
    for (i64 base = 0; base < nb; base += SCAN_THREADS) {
        const i64 i = base + threadIdx.x;
        const i64 v = i < nb ? sums[i] : 0;
        i64 total;
        const i64 ex = block_exclusive_scan(v, sh, &total);
        if (i < nb) sums[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) *grand_total = carry;
}

__global__ void k_scan_tiles(const i64* in, i64* out, i64 n, const i64* offsets) {
    __shared__ i64 sh[SCAN_THREADS / 32];
    const i64 base = i64(blockIdx.x) * SCAN_TILE;
    i64 v[SCAN_ITEMS];
    i64 s = 0;
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const i64 i = base + i64(threadIdx.x) * SCAN_ITEMS + k;
        v[k] = i < n ? in[i] : 0;
        s += v[k];
    }
    i64 run = block_exclusive_scan(s, sh, nullptr) + offsets[blockIdx.x];
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const i64 i = base + i64(threadIdx.x) * SCAN_ITEMS + k;
        if (i < n) out[i] = run;
        run += v[k];
    }
}

}  // namespace

void exclusive_scan(Ctx& ctx, const i64* in, i64* out, i64 n, i64* total_host) {
    const i64 nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    ctx.i64_scratch_a.reserve(size_t(nb + 2));
    i64* sums = ctx.i64_scratch_a.p;
    i64* grand = sums + nb + 1;
    if (n > 0) {
        NL_LAUNCH(k_tile_sums, unsigned(nb), SCAN_THREADS, 0, ctx.stream, in, n, sums);
        NL_LAUNCH(k_scan_sums, 1, SCAN_THREADS, 0, ctx.stream, sums, nb, grand);
        NL_LAUNCH(k_scan_tiles, unsigned(nb), SCAN_THREADS, 0, ctx.stream, in, out, n, sums);
    } else {
        NL_CUDA(cudaMemsetAsync(grand, 0, sizeof(i64), ctx.stream));
    }
    if (total_host) {
        NL_CUDA(cudaMemcpyAsync(total_host, grand, sizeof(i64), cudaMemcpyDeviceToHost, ctx.stream));
        NL_CUDA(cudaStreamSynchronize(ctx.stream));
    }
}

i64 device_read_i64(Ctx& ctx, const i64* p) {
    i64 v = 0;
    NL_CUDA(cudaMemcpyAsync(&v, p, sizeof(i64), cudaMemcpyDeviceToHost, ctx.stream));
    NL_CUDA(cudaStreamSynchronize(ctx.stream));
    return v;
}

}  // namespace nlgpu
