// noalloc.cu — candidate-pair generation for callers that cannot allocate
// device memory.
//
// Some callers of this library may not call cudaMalloc at the point where
// they need the broadphase: code running inside another framework's memory
// pool or allocator (which owns all device memory and forbids side
// allocations), real-time loops that must not hit the driver's allocator, or
// plugins that are handed pre-allocated input/output buffers and nothing
// else.  cpgpu_pairs_noalloc serves them: the caller passes the AABBs and the
// output buffers (device memory it already owns) and the call allocates
// nothing.  Its only scratch (per-body overlap counts, and a grid's buckets) is
// a file-scope __device__ array of fixed size, so the maximum body count per
// call is kNoAllocMaxBodies.
//
// Same result as the batch path's pair generation (broadphase.cu): every pair
// (i, j), i < j, whose AABBs overlap under the inclusive test, in (i, j)
// order, ids 1-based.
//
// Up to kNoAllocBrute boxes a warp tests each box against all later ones, 32 at
// a time (n^2 / 2 tests).  Above, the boxes go into a hashed grid and a warp
// tests a box against those of its 27 cells.
#include <cstdio>
#include <mutex>
#include <vector>

#include "kernels.cuh"
#include "pairs.cuh"

extern "C" {
#include "../../include/cpgpu.h"
}

namespace cpgpu {

constexpr int kNoAllocMaxBodies = 1 << 16;
// the pass over all later boxes up to here, the grid above: 40 us against 51 at
// 4,096 boxes, 91 against 67 at 8,192 (4.7 ms against 0.2 at 65,536)
constexpr int kNoAllocBrute = 5120;
constexpr int kNoAllocBuckets = 1 << 15;

// Scratch of every call on a device: per-body overlap counts (turned into
// output offsets in place), bucket starts, the boxes by bucket, the boxes that
// do not go into the grid, and the grid's numbers.  Every GPU that loads the
// library holds it (about 650 KB) until the process exits.
struct NoAllocScratch {
    int count[kNoAllocMaxBodies];
    int bucket[kNoAllocBuckets];
    int chunk[kNoAllocMaxBodies / 1024];  // overlaps per 1,024 boxes
    uint16_t ids[kNoAllocMaxBodies];
    uint16_t far_ids[kNoAllocMaxBodies];
    int n_far, total;
    float inv;
};
static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

namespace {

struct NaLoad {
    const float2* b;   // boxes of 6 floats, 8-byte aligned at the least
    const float* f;
    bool vec;
    __device__ __forceinline__ explicit NaLoad(const float* aabbs)
        : b(reinterpret_cast<const float2*>(aabbs)), f(aabbs), vec((reinterpret_cast<uintptr_t>(aabbs) & 7) == 0) {}
    __device__ __forceinline__ PairBox operator()(int j) const {
        if (vec) {
            const float2 x = b[3 * j], y = b[3 * j + 1], z = b[3 * j + 2];
            return PairBox{x.x, x.y, y.x, y.y, z.x, z.y};
        }
        const float* p = f + 6 * j;
        return PairBox{p[0], p[1], p[2], p[3], p[4], p[5]};
    }
};
struct NaEnd {
    int n;
    __device__ __forceinline__ int operator()(int) const { return n; }
};
__device__ __forceinline__ void na_put(uint32_t* pairs, int cap, int o, int i, int j) {
    if ((unsigned)o < (unsigned)cap) { pairs[2 * (size_t)o] = (uint32_t)i + 1; pairs[2 * (size_t)o + 1] = (uint32_t)j + 1; }
}

__global__ void __launch_bounds__(256) k_na_count(const float* aabbs, int n, NoAllocScratch* s) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    int c[1];
    pairs_of_group<1>(i, n, NaLoad(aabbs), NaEnd{n}, [](int, int, int) {}, c);
    if ((threadIdx.x & 31) == 0) s->count[i] = c[0];
}
__global__ void __launch_bounds__(1024) k_na_scan(int n, NoAllocScratch* s, int* count) {
    const int total = block_prefix_1024(s->count, n);
    if (threadIdx.x == 0) { *count = total; s->total = total; }
}
__global__ void __launch_bounds__(256) k_na_write(const float* aabbs, int n, const NoAllocScratch* s, uint32_t* pairs, int cap) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    const int o = s->count[i];
    int c[1];
    pairs_of_group<1>(i, n, NaLoad(aabbs), NaEnd{n}, [&](int, int j, int k) { na_put(pairs, cap, o + k, i, j); }, c);
}

// ---- the grid ------------------------------------------------------------------------
__device__ __forceinline__ PairGrid<uint16_t> na_grid(NoAllocScratch* s, int n) {
    return PairGrid<uint16_t>{s->bucket, s->ids, s->far_ids, &s->n_far, &s->inv, kNoAllocBuckets, n, kNoAllocMaxBodies};
}
struct NaWorld {   // one world
    __device__ __forceinline__ int operator()(int) const { return 0; }
};
__global__ void __launch_bounds__(1024) k_na_begin(const float* aabbs, int n, NoAllocScratch* s) {
    if (blockIdx.x == 0 && threadIdx.x < kNoAllocMaxBodies / 1024) s->chunk[threadIdx.x] = 0;
    const int step = grid_sample_step(n);
    grid_begin(na_grid(s, n), grid_sample_count(n), NaLoad(aabbs), [=](int k) { return k * step; });
}
__global__ void __launch_bounds__(256) k_na_put(const float* aabbs, int n, NoAllocScratch* s, int pass) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) grid_put(na_grid(s, n), i, 0, NaLoad(aabbs), pass);
}
__global__ void __launch_bounds__(1024) k_na_buckets(NoAllocScratch* s) { block_prefix_1024(s->bucket, kNoAllocBuckets); }
__global__ void __launch_bounds__(256) k_na_grid_count(const float* aabbs, int n, NoAllocScratch* s) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    const NaLoad load(aabbs);
    int c = grid_near(na_grid(s, n), i, 0, load, NaWorld{}, [](int) {});
    if (c == -2) return;   // k_na_far's
    if (c < 0) {
        int one[1];
        pairs_of_group<1>(i, n, load, NaEnd{n}, [](int, int, int) {}, one);
        c = one[0];
    }
    if ((threadIdx.x & 31) == 0) {
        s->count[i] = c;
        if (c > 0) atomicAdd(&s->chunk[i >> 10], c);
    }
}
__global__ void __launch_bounds__(1024) k_na_far(const float* aabbs, int n, NoAllocScratch* s, uint32_t* pairs, int cap, int write) {
    // one thread reads for the block: its threads go through the same barriers
    // whatever another call writes meanwhile
    __shared__ int sh_m, sh_i;
    if (threadIdx.x == 0) sh_m = min(s->n_far, kNoAllocMaxBodies);
    __syncthreads();
    const int m = sh_m;
    for (int k = blockIdx.x; k < m; k += gridDim.x) {
        if (threadIdx.x == 0) sh_i = min((int)s->far_ids[k], n - 1);
        __syncthreads();
        const int i = sh_i, o = write ? s->count[i] : 0;
        const int c = grid_far(i, n, NaLoad(aabbs), write != 0, [&](int r, int j) { na_put(pairs, cap, o + r, i, j); });
        if (!write && threadIdx.x == 0) {
            s->count[i] = c;
            if (c > 0) atomicAdd(&s->chunk[i >> 10], c);
        }
    }
}
// counts to offsets, a block per 1,024 boxes: every block sums the chunks
// before its own (at most 64)
__global__ void __launch_bounds__(1024) k_na_offsets(int n, NoAllocScratch* s, int* count) {
    __shared__ int ws[32], before;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, i = blockIdx.x * 1024 + t;
    if (wid == 0) {
        int x = 0, all = 0;
        for (int k = lane; k < (int)gridDim.x; k += 32) { all += s->chunk[k]; if (k < (int)blockIdx.x) x += s->chunk[k]; }
        x = __reduce_add_sync(0xffffffffu, x);
        all = __reduce_add_sync(0xffffffffu, all);
        if (lane == 0) {
            before = x;
            if (blockIdx.x == 0) { *count = all; s->total = all; }
        }
    }
    const int v = i < n ? s->count[i] : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) { const int q = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += q; }
    if (lane == 31) ws[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int y = ws[lane];
        for (int o = 1; o < 32; o <<= 1) { const int q = __shfl_up_sync(0xffffffffu, y, o); if (lane >= o) y += q; }
        ws[lane] = y;
    }
    __syncthreads();
    if (i < n) s->count[i] = before + x - v + (wid > 0 ? ws[wid - 1] : 0);
}
__global__ void __launch_bounds__(256) k_na_grid_write(const float* aabbs, int n, NoAllocScratch* s, uint32_t* pairs, int cap) {
    __shared__ int near[8][kGridNear], n_near[8];
    const int wid = threadIdx.x >> 5, i = blockIdx.x * 8 + wid;
    if (i >= n) return;
    const int o = __shfl_sync(0xffffffffu, s->count[i], 0);
    const int m = __shfl_sync(0xffffffffu, i + 1 < n ? s->count[i + 1] : s->total, 0) - o;
    if (m == 0 || o >= cap) return;
    grid_write(na_grid(s, n), i, n, m, NaLoad(aabbs), NaWorld{}, NaEnd{n}, near[wid], &n_near[wid],
               [&](int k, int j) { na_put(pairs, cap, o + k, i, j); });
}

// Device address of the scratch array, looked up with the device current
// (host code must not use the symbol itself as a pointer).  The address is
// cached per CUDA context, identified by the driver's context id, so that a
// caller who resets the device (a new primary context, the module loaded
// again) gets the new address instead of a stale one.  If the driver entry
// points for the context id are unavailable, the address is looked up again
// on every call.
typedef int (*CtxGetCurrentFn)(void**);
typedef int (*CtxGetIdFn)(void*, unsigned long long*);
struct NaCache { unsigned long long ctx_id; NoAllocScratch* ptr; };
std::mutex g_na_mutex;
std::vector<NaCache> g_na_cache;
CtxGetCurrentFn g_ctx_current = nullptr;
CtxGetIdFn g_ctx_id = nullptr;
bool g_ctx_fns_looked_up = false;

bool current_context_id(unsigned long long* id) {
    if (!g_ctx_fns_looked_up) {
        g_ctx_fns_looked_up = true;
        cudaDriverEntryPointQueryResult q1, q2;
        void *f1 = nullptr, *f2 = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1) == cudaSuccess &&
            cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2) == cudaSuccess &&
            q1 == cudaDriverEntryPointSuccess && q2 == cudaDriverEntryPointSuccess && f1 && f2) {
            g_ctx_current = reinterpret_cast<CtxGetCurrentFn>(f1);
            g_ctx_id = reinterpret_cast<CtxGetIdFn>(f2);
        }
    }
    if (!g_ctx_current || !g_ctx_id) return false;
    void* ctx = nullptr;
    if (g_ctx_current(&ctx) != 0 || !ctx) return false;
    return g_ctx_id(ctx, id) == 0;
}

int scratch_for_current_device(NoAllocScratch** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return CPGPU_ERR_NO_DEVICE;
    std::lock_guard<std::mutex> lock(g_na_mutex);
    unsigned long long id = 0;
    if (current_context_id(&id))
        for (const NaCache& c : g_na_cache)
            if (c.ctx_id == id) { *out = c.ptr; return CPGPU_OK; }
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess) return CPGPU_ERR_CUDA;
    // the lookup made the device's primary context current if it was not
    if (current_context_id(&id)) g_na_cache.push_back({id, static_cast<NoAllocScratch*>(p)});
    *out = static_cast<NoAllocScratch*>(p);
    return CPGPU_OK;
}

}  // namespace
}  // namespace cpgpu

extern "C" int cpgpu_pairs_noalloc(const float* aabbs, int n_bodies, uint32_t* pairs, int cap, int* count, void* stream) {
    using namespace cpgpu;
    if (n_bodies < 0 || cap < 0 || !count || (n_bodies > 0 && !aabbs) || (cap > 0 && !pairs)) {
        set_last_error("cpgpu_pairs_noalloc: null buffer or negative size");
        return CPGPU_ERR_INVALID_ARG;
    }
    if (n_bodies > kNoAllocMaxBodies) {
        set_last_error("cpgpu_pairs_noalloc: more than 65536 bodies (the fixed scratch holds one count per body)");
        return CPGPU_ERR_INVALID_ARG;
    }
    // an error left by earlier work on this thread is not ours to report or
    // to clear: refuse to run and leave it pending for its owner
    cudaError_t pending = cudaPeekAtLastError();
    if (pending != cudaSuccess) {
        char msg[256];
        std::snprintf(msg, sizeof msg, "cpgpu_pairs_noalloc: an earlier CUDA error is pending (%s); nothing launched",
                      cudaGetErrorName(pending));
        set_last_error(msg);
        return CPGPU_ERR_CUDA;
    }
    NoAllocScratch* scratch = nullptr;
    int rc = scratch_for_current_device(&scratch);
    if (rc != CPGPU_OK) {
        set_last_error("cpgpu_pairs_noalloc: no usable CUDA device or scratch symbol lookup failed");
        return rc;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int warps = (n_bodies + 7) / 8;
    if (n_bodies <= kNoAllocBrute) {
        if (n_bodies > 0) k_na_count<<<warps, 256, 0, st>>>(aabbs, n_bodies, scratch);
        k_na_scan<<<1, 1024, 0, st>>>(n_bodies, scratch, count);
        if (n_bodies > 0) k_na_write<<<warps, 256, 0, st>>>(aabbs, n_bodies, scratch, pairs, cap);
    } else {
        const int per = (n_bodies + 255) / 256;
        k_na_begin<<<17, 1024, 0, st>>>(aabbs, n_bodies, scratch);
        k_na_put<<<per, 256, 0, st>>>(aabbs, n_bodies, scratch, 0);
        k_na_buckets<<<1, 1024, 0, st>>>(scratch);
        k_na_put<<<per, 256, 0, st>>>(aabbs, n_bodies, scratch, 1);
        k_na_grid_count<<<warps, 256, 0, st>>>(aabbs, n_bodies, scratch);
        k_na_far<<<64, 1024, 0, st>>>(aabbs, n_bodies, scratch, pairs, cap, 0);
        k_na_offsets<<<(n_bodies + 1023) / 1024, 1024, 0, st>>>(n_bodies, scratch, count);
        k_na_far<<<64, 1024, 0, st>>>(aabbs, n_bodies, scratch, pairs, cap, 1);
        k_na_grid_write<<<warps, 256, 0, st>>>(aabbs, n_bodies, scratch, pairs, cap);
    }
    if (cudaGetLastError() != cudaSuccess) {
        set_last_error("cpgpu_pairs_noalloc: kernel launch failed");
        return CPGPU_ERR_CUDA;
    }
    return CPGPU_OK;
}
