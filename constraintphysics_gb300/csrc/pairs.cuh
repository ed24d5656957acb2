// pairs.cuh — candidate pairs of axis-aligned boxes, shared by the batch's pair
// generation (broadphase.cu) and the allocation-free one (noalloc.cu): a group
// of boxes tested by one warp against all later ones, and a hashed grid for
// many boxes.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "gridsample.h"

namespace cpgpu {

// Boxes a warp tests together: each later box is loaded once for all of them.
constexpr int kPairGroup = 4;

struct PairBox { float lx, ly, lz, hx, hy, hz; };

// inclusive overlap (AABB::intersects, AABB.h:10-14); comparisons with NaN are
// false, so a NaN coordinate separates nothing
__device__ __forceinline__ bool box_meet(const PairBox& a, const PairBox& b) {
    return !(a.hx < b.lx || a.lx > b.hx || a.hy < b.ly || a.ly > b.hy || a.hz < b.lz || a.lz > b.hz);
}

// For the boxes i0 .. i0 + G - 1 (those below `n`): every overlapping j > i below
// end(i), j ascending.  load(j) gives a box, end(i) the box's exclusive bound
// (ascending over the group); hit(g, j, k) is called by the lane that holds the
// k-th overlap of box i0 + g, counted from 0.  Every lane returns the counts.
template <int G, class Load, class End, class Hit>
__device__ __forceinline__ void pairs_of_group(int i0, int n, const Load& load, const End& end, const Hit& hit, int cnt[G]) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    PairBox a[G];
    int e[G];
#pragma unroll
    for (int g = 0; g < G; g++) {
        const int i = i0 + g;
        e[g] = i < n ? end(i) : 0;
        if (i < n) a[g] = load(i);
        cnt[g] = 0;
    }
    int last = 0;
#pragma unroll
    for (int g = 0; g < G; g++) last = max(last, e[g]);
    // the next 32 boxes are loaded while these are tested: with few warps the
    // pass is bound by that latency
    PairBox b{}, nx{};
    if (i0 + 1 + lane < last) b = load(i0 + 1 + lane);
    for (int j0 = i0 + 1; j0 < last; j0 += 32) {
        const int j = j0 + lane;
        if (j + 32 < last) nx = load(j + 32);
#pragma unroll
        for (int g = 0; g < G; g++) {
            const bool h = j > i0 + g && j < e[g] && box_meet(a[g], b);
            const unsigned m = __ballot_sync(0xffffffffu, h);
            if (h) hit(g, j, cnt[g] + __popc(m & below));
            cnt[g] += __popc(m);
        }
        b = nx;
    }
}

// exclusive prefix of v[0 .. n) in place by one block of 1,024 threads, each
// taking a contiguous run; returns the total to every thread
__device__ __forceinline__ int block_prefix_1024(int* v, int n) {
    __shared__ int ws[33];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int per = ((n + 1023) / 1024 + 3) & ~3;   // a multiple of 4, so that runs start 16-byte aligned
    const int b = min(n, tid * per), e = min(n, b + per);
    int s = 0;
    int k = b;
    for (; k + 4 <= e; k += 4) { const int4 q = *reinterpret_cast<const int4*>(v + k); s += q.x + q.y + q.z + q.w; }
    for (; k < e; k++) s += v[k];
    int x = s;
    for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += t; }
    if (lane == 31) ws[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int y = ws[lane];
        for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, y, o); if (lane >= o) y += t; }
        ws[lane] = y;
    }
    __syncthreads();
    int run = x - s + (wid > 0 ? ws[wid - 1] : 0);
    const int total = ws[31];
    for (k = b; k + 4 <= e; k += 4) {
        int4 q = *reinterpret_cast<const int4*>(v + k);
        const int4 o = make_int4(run, run + q.x, run + q.x + q.y, run + q.x + q.y + q.z);
        run = o.w + q.w;
        *reinterpret_cast<int4*>(v + k) = o;
    }
    for (; k < e; k++) { const int t = v[k]; v[k] = run; run += t; }
    return total;
}

// ---- many boxes: a grid of cells hashed into buckets -----------------------------
// A box that reaches at most one cell beyond the cell of its lower corner meets
// only boxes of the 27 cells around it; the others (larger, NaN, inverted or
// out of the cell numbers' range) are listed apart and tested against all.
// Cell numbers come from the same rounded products everywhere, which are
// monotonic in the coordinate, so no neighbour is missed; the result does not
// depend on the cells at all.  The bucket hash takes the primes of Teschner et
// al. ("Optimized Spatial Hashing for Collision Detection of Deformable
// Objects", 2003) and, for the world, Knuth's multiplier.
// Nothing read from the grid's own arrays is used as an index unchecked: the
// allocation-free call's are shared by all calls on a device, and calls that
// overlap (which gives wrong pairs) still stay inside their buffers.
template <class Id>
struct PairGrid {
    int* bucket;       // [buckets]: sizes, their exclusive prefix, then (filled) each bucket's end
    Id* ids;           // the boxes by bucket
    Id* far_ids;       // the boxes outside the grid
    int* n_far;
    float* inv;        // 1 / cell side (0: no usable box)
    int buckets;       // a power of two
    int n, cap;        // boxes; entries of ids and far_ids
    __device__ __forceinline__ int of(int x, int y, int z, int w) const {
        return (int)(((uint32_t)x * 73856093u ^ (uint32_t)y * 19349663u ^ (uint32_t)z * 83492791u ^ (uint32_t)w * 2654435761u) &
                     (uint32_t)(buckets - 1));
    }
};
struct PairCell { int x, y, z; };
__device__ __forceinline__ bool box_plain(const PairBox& b) {   // finite, not inverted
    const float lim = 1e30f;
    return b.lx <= b.hx && b.ly <= b.hy && b.lz <= b.hz && b.lx > -lim && b.ly > -lim && b.lz > -lim && b.hx < lim && b.hy < lim &&
           b.hz < lim;
}
__device__ __forceinline__ bool box_cell(const PairBox& b, float inv, PairCell* c) {
    if (!(inv > 0.f) || !box_plain(b)) return false;
    const float x = floorf(__fmul_rn(b.lx, inv)), y = floorf(__fmul_rn(b.ly, inv)), z = floorf(__fmul_rn(b.lz, inv));
    const float lim = 1e6f;
    if (!(fabsf(x) < lim && fabsf(y) < lim && fabsf(z) < lim)) return false;
    if (floorf(__fmul_rn(b.hx, inv)) - x > 1.f || floorf(__fmul_rn(b.hy, inv)) - y > 1.f || floorf(__fmul_rn(b.hz, inv)) - z > 1.f)
        return false;
    *c = PairCell{(int)x, (int)y, (int)z};
    return true;
}

// The first block (1,024 threads) sizes the cells from the sampled boxes (at most
// kGridSamples; sample(k): the k-th), the others empty the buckets.  A cell is as
// wide as the widest box within three times the mean: those boxes are all in
// the grid (a few hundred outside cost every warp a walk over them: on 20,000
// mixed bodies 0.48 ms with cells of 1.25 times the mean).
template <class Id, class Load, class Sample>
__device__ __forceinline__ void grid_begin(const PairGrid<Id>& g, int samples, const Load& load, const Sample& sample) {
    if (blockIdx.x > 0) {
        for (int i = (blockIdx.x - 1) * blockDim.x + threadIdx.x; i < g.buckets; i += (gridDim.x - 1) * blockDim.x) g.bucket[i] = 0;
        return;
    }
    __shared__ float ss[32];
    __shared__ int sm[32];
    constexpr int kPer = kGridSamples / 1024;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float ext[kPer], sum = 0.f;
    int m = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const int q = threadIdx.x + 1024 * k;
        ext[k] = -1.f;
        if (q < samples) {
            const PairBox b = load(sample(q));
            const float e = fmaxf(b.hx - b.lx, fmaxf(b.hy - b.ly, b.hz - b.lz));
            if (box_plain(b) && e < 1e15f) { ext[k] = e; sum += e; m++; }
        }
    }
    for (int o = 16; o > 0; o >>= 1) { sum += __shfl_xor_sync(0xffffffffu, sum, o); m += __shfl_xor_sync(0xffffffffu, m, o); }
    if (lane == 0) { ss[wid] = sum; sm[wid] = m; }
    __syncthreads();
    sum = 0.f;
    m = 0;
    for (int q = 0; q < 32; q++) { sum += ss[q]; m += sm[q]; }
    const float cap = m > 0 ? 3.f * sum / (float)m : 0.f;
    float top = 0.f;
#pragma unroll
    for (int k = 0; k < kPer; k++) if (ext[k] <= cap) top = fmaxf(top, ext[k]);
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    __syncthreads();
    if (lane == 0) ss[wid] = top;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 0; q < 32; q++) top = fmaxf(top, ss[q]);
        *g.inv = top > 1e-15f ? 0.999f / top : 0.f;
        *g.n_far = 0;
    }
}
// box i into its bucket: pass 0 counts, pass 1 (after the prefix) stores it
template <class Id, class Load>
__device__ __forceinline__ void grid_put(const PairGrid<Id>& g, int i, int w, const Load& load, int pass) {
    PairCell c;
    if (box_cell(load(i), *g.inv, &c)) {
        const int b = g.of(c.x, c.y, c.z, w);
        const int at = atomicAdd(&g.bucket[b], 1);
        if (pass == 1 && (unsigned)at < (unsigned)g.cap) g.ids[at] = (Id)i;
    } else if (pass == 0) {
        const int at = atomicAdd(g.n_far, 1);
        if ((unsigned)at < (unsigned)g.cap) g.far_ids[at] = (Id)i;
    }
}
// Box i's overlaps j > i in its world w by one warp, in no order: lane k < 27
// walks the bucket of one neighbouring cell (boxes of other cells or worlds in
// it are passed over, so cells that share a bucket give nothing twice), then
// the lanes share the boxes outside the grid.  hit(j) is called for each.
// Returns the count to every lane; -1 (nothing called): it has too many
// candidates to walk this way; -2: it is outside the grid.
constexpr int kGridMost = 64, kGridFar = 2048;
template <class Id, class Load, class World, class Hit>
__device__ __forceinline__ int grid_near(const PairGrid<Id>& g, int i, int w, const Load& load, const World& world, const Hit& hit) {
    const int lane = threadIdx.x & 31;
    const PairBox a = load(i);
    const float inv = __shfl_sync(0xffffffffu, *g.inv, 0);   // one value for the warp's branches
    PairCell c;
    if (!box_cell(a, inv, &c)) return -2;
    int b0 = 0, b1 = 0, x = 0, y = 0, z = 0;
    if (lane < 27) {
        x = c.x + lane % 3 - 1;
        y = c.y + lane / 3 % 3 - 1;
        z = c.z + lane / 9 - 1;
        const int b = g.of(x, y, z, w);
        b0 = b > 0 ? max(g.bucket[b - 1], 0) : 0;
        b1 = min(g.bucket[b], g.cap);
    }
    const int n_far = min(*g.n_far, g.cap);
    if (__any_sync(0xffffffffu, b1 - b0 > kGridMost) || n_far > kGridFar) return -1;
    int cnt = 0;
#pragma unroll 4
    for (int k = b0; k < b1; k++) {
        const int j = g.ids[k];
        if (j <= i || j >= g.n || world(j) != w) continue;
        const PairBox b = load(j);
        PairCell cj;
        if (box_meet(a, b) && box_cell(b, inv, &cj) && cj.x == x && cj.y == y && cj.z == z) { hit(j); cnt++; }
    }
    for (int k = lane; k < n_far; k += 32) {
        const int j = g.far_ids[k];
        if (j > i && j < g.n && world(j) == w && box_meet(a, load(j))) { hit(j); cnt++; }
    }
    return __reduce_add_sync(0xffffffffu, cnt);
}
// Box i's `m` overlaps, written by one warp in ascending order: put(k, j).
// `near`: the warp's kGridNear entries of shared memory, `n_near` its counter.
// (A box outside the grid is grid_far's.)
constexpr int kGridNear = 256;
template <class Id, class Load, class World, class End, class Put>
__device__ __forceinline__ void grid_write(const PairGrid<Id>& g, int i, int n, int m, const Load& load, const World& world,
                                           const End& end, int* near, int* n_near, const Put& put) {
    const int lane = threadIdx.x & 31;
    PairCell cell;
    if (!box_cell(load(i), __shfl_sync(0xffffffffu, *g.inv, 0), &cell)) return;
    if (lane == 0) *n_near = 0;
    __syncwarp();
    const auto keep = [&](int j) {
        const int at = atomicAdd(n_near, 1);
        if (at < kGridNear) near[at] = j;
    };
    const int c = m <= kGridNear ? min(grid_near(g, i, world(i), load, world, keep), kGridNear) : -1;
    __syncwarp();
    if (c >= 0) {
        for (int k = lane; k < c; k += 32) {   // each overlap at its rank
            int r = 0;
            const int j = near[k];
            for (int q = 0; q < c; q++) r += near[q] < j;
            put(r, j);
        }
    } else {
        int one[1];
        pairs_of_group<1>(i, n, load, end, [&](int, int j, int k) { put(k, j); }, one);
    }
}
// A box outside the grid against every later one below `e`, by one block (a
// warp alone takes 180 us over 20,000 boxes): each warp a run of the range.
// Returns the count to every thread; `write`: put(k, j) in ascending order.
template <class Load, class Put>
__device__ __forceinline__ int grid_far(int i, int e, const Load& load, bool write, const Put& put) {
    __shared__ int sums[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const PairBox a = load(i);
    const int per = ((e - i - 1 + nw - 1) / nw + 31) & ~31;
    const int b0 = i + 1 + wid * per, b1 = min(e, b0 + per);
    int c = 0;
    for (int j0 = b0; j0 < b1; j0 += 32) c += __popc(__ballot_sync(0xffffffffu, j0 + lane < b1 && box_meet(a, load(min(j0 + lane, e - 1)))));
    if (lane == 0) sums[wid] = c;
    __syncthreads();
    int base = 0, total = 0;
    for (int q = 0; q < nw; q++) {
        if (q < wid) base += sums[q];
        total += sums[q];
    }
    if (write)
        for (int j0 = b0; j0 < b1; j0 += 32) {
            const bool h = j0 + lane < b1 && box_meet(a, load(min(j0 + lane, e - 1)));
            const unsigned m = __ballot_sync(0xffffffffu, h);
            if (h) put(base + __popc(m & below), j0 + lane);
            base += __popc(m);
        }
    __syncthreads();
    return total;
}

}  // namespace cpgpu
