// broadphase.cu — gravity, candidate pairs and the geometry/AABB update.
//
// Pair generation returns exactly the set the reference's AABB tree returns:
// every pair of bodies of the same world whose true AABBs overlap under the
// inclusive test of AABB::intersects (ConstraintPhysics/src/AABB.h:10-14; the
// tree query AABB_Tree.h:153-224 visits every overlapping leaf pair once).
// Pairs are emitted as (lower id, higher id) sorted by (a, b): a warp counts the
// overlaps of kPairGroup consecutive bodies with the later bodies of their
// world, 32 of those at a time, an exclusive scan gives each body its output
// offset, and a second pass writes.  Bound by the tests' FP32 issue in large
// worlds and by latency in small ones; a thread per body (each walking the
// rest of its world alone) took 117 us a pass on one world of 1,000 bodies
// where this takes 12.  The bodies of worlds above kTileWorld bodies go into a
// hashed grid instead (pairs.cuh).
#include <algorithm>

#include "kernels.cuh"
#include "devmath.cuh"
#include "pairs.cuh"
#include "scan.cuh"
#include "shapes.cuh"

namespace cpgpu {

namespace {
__global__ void k_gravity(Dev d) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.n_bodies; i += gridDim.x * blockDim.x) {
        if (d.movement[i] != 0) continue;
        const WorldParams& p = d.wparams[d.world[i]];
        float4 v = d.vel[i];
        // vel += gravity * step_time (PhysicsEngine.cpp:85)
        v.x += p.gx * p.dt; v.y += p.gy * p.dt; v.z += p.gz * p.dt;
        d.vel[i] = v;
    }
}

struct BodyBox {
    const float4 *lo, *hi;
    __device__ __forceinline__ PairBox operator()(int j) const {
        const float4 l = lo[j], h = hi[j];
        return PairBox{l.x, l.y, l.z, h.x, h.y, h.z};
    }
};
__global__ void __launch_bounds__(256) k_pairs(Dev d, int write) {
    const int nw = gridDim.x * (blockDim.x >> 5);
    const bool big = d.grid_buckets > 0;   // the batch holds worlds of the grid
    const BodyBox load{d.aabb_lo, d.aabb_hi};
    auto end = [&](int i) {
        const int w = d.world[i], e = d.world_start[w + 1];
        return big && e - d.world_start[w] > kTileWorld ? 0 : e;
    };
    for (int i0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kPairGroup; i0 < d.n_bodies; i0 += nw * kPairGroup) {
        int c[kPairGroup];
        if (!write) {
            pairs_of_group<kPairGroup>(i0, d.n_bodies, load, end, [](int, int, int) {}, c);
            if ((threadIdx.x & 31) == 0)
#pragma unroll
                for (int g = 0; g < kPairGroup; g++)
                    if (i0 + g < d.n_bodies && !(big && end(i0 + g) == 0)) d.pair_count[i0 + g] = c[g];
        } else {
            int o[kPairGroup];
#pragma unroll
            for (int g = 0; g < kPairGroup; g++) o[g] = i0 + g < d.n_bodies ? d.pair_count[i0 + g] : 0;
            pairs_of_group<kPairGroup>(i0, d.n_bodies, load, end, [&](int g, int j, int k) {
                int at = o[0];
#pragma unroll
                for (int q = 1; q < kPairGroup; q++) at = g == q ? o[q] : at;
                at += k;
                if (at < d.cap_pairs) { d.pair_a[at] = i0 + g; d.pair_b[at] = j; }
            }, c);
        }
    }
}

// Large worlds: their bodies go into one hashed grid (keyed by the world too),
// and a warp tests a body against those of its 27 cells.
struct GridWorld {
    const Dev& d;
    __device__ __forceinline__ int operator()(int i) const { return d.world[i]; }
};
__device__ __forceinline__ PairGrid<int> dev_grid(const Dev& d) {
    return PairGrid<int>{d.grid_bucket, d.grid_ids, d.grid_far, d.grid_n_far, d.grid_inv, d.grid_buckets, d.n_bodies, d.n_bodies};
}
__device__ __forceinline__ bool in_grid_world(const Dev& d, int i) {
    const int w = d.world[i];
    return d.world_start[w + 1] - d.world_start[w] > kTileWorld;
}
__global__ void __launch_bounds__(1024) k_grid_begin(Dev d) {
    grid_begin(dev_grid(d), d.n_grid_sample, BodyBox{d.aabb_lo, d.aabb_hi}, [&](int k) { return d.grid_sample[k]; });
}
__global__ void __launch_bounds__(256) k_grid_put(Dev d, int pass) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.n_bodies; i += gridDim.x * blockDim.x)
        if (in_grid_world(d, i)) grid_put(dev_grid(d), i, d.world[i], BodyBox{d.aabb_lo, d.aabb_hi}, pass);
}
__global__ void __launch_bounds__(1024) k_grid_buckets(Dev d) { block_prefix_1024(d.grid_bucket, d.grid_buckets); }
__global__ void __launch_bounds__(256) k_grid_count(Dev d) {
    const BodyBox load{d.aabb_lo, d.aabb_hi};
    for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < d.n_bodies; i += gridDim.x * 8) {
        if (!in_grid_world(d, i)) continue;
        const int w = d.world[i];
        int c = grid_near(dev_grid(d), i, w, load, GridWorld{d}, [](int) {});
        if (c == -2) continue;   // k_grid_far's
        if (c < 0) {
            int one[1];
            pairs_of_group<1>(i, d.n_bodies, load, [&](int) { return d.world_start[w + 1]; }, [](int, int, int) {}, one);
            c = one[0];
        }
        if ((threadIdx.x & 31) == 0) d.pair_count[i] = c;
    }
}
__global__ void __launch_bounds__(1024) k_grid_far(Dev d, int write) {
    const int m = *d.grid_n_far;
    for (int k = blockIdx.x; k < m; k += gridDim.x) {
        const int i = d.grid_far[k], o = write ? d.pair_count[i] : 0;
        const int c = grid_far(i, d.world_start[d.world[i] + 1], BodyBox{d.aabb_lo, d.aabb_hi}, write != 0, [&](int r, int j) {
            if (o + r < d.cap_pairs) { d.pair_a[o + r] = i; d.pair_b[o + r] = j; }
        });
        if (!write && threadIdx.x == 0) d.pair_count[i] = c;
    }
}
__global__ void __launch_bounds__(256) k_grid_write(Dev d) {
    __shared__ int near[8][kGridNear], n_near[8];
    const int wid = threadIdx.x >> 5;
    const BodyBox load{d.aabb_lo, d.aabb_hi};
    for (int i = blockIdx.x * 8 + wid; i < d.n_bodies; i += gridDim.x * 8) {
        if (!in_grid_world(d, i)) continue;
        const int o = d.pair_count[i], m = (i + 1 < d.n_bodies ? d.pair_count[i + 1] : *d.n_pairs) - o;
        if (m == 0 || o >= d.cap_pairs) continue;
        const int e = d.world_start[d.world[i] + 1];
        grid_write(dev_grid(d), i, d.n_bodies, m, load, GridWorld{d}, [&](int) { return e; }, near[wid], &n_near[wid],
                   [&](int k, int j) { if (o + k < d.cap_pairs) { d.pair_a[o + k] = i; d.pair_b[o + k] = j; } });
    }
}

// pair counts to offsets; the total is clamped to the capacity, and this
// step's narrowphase counters start at zero
struct PairScan {
    static __device__ int in(const Dev& d, int i) { return d.pair_count[i]; }
    static __device__ void out(const Dev& d, int i, int x) { d.pair_count[i] = x; }
    static __device__ void done(const Dev& d, int total) {
        if (total > d.cap_pairs) { atomicOr(d.status, ST_PAIR_OVERFLOW); total = d.cap_pairs; }
        *d.n_pairs = total;
        if (d.has_mesh || d.has_union) *d.mm_count = 0;   // mesh store of this step's narrowphase
        d.np_next[0] = d.np_next[1] = 0;
        for (int k = 0; k < 32; k++) d.prim_count_k[k] = 0;
    }
};

// RigidBody::updateGeometry (RigidBody.cpp:281-312) for moved bodies: the
// orientation is renormalised and the AABB recomputed from the world geometry
// (gen_AABB of the body's primitive).  `mode` 2 (a batch's first pass): every
// body's AABB, the orientations flagged in `moved` (poses set through the
// API) renormalised.
__global__ void k_geometry(Dev d, int mode) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.n_bodies; i += gridDim.x * blockDim.x) {
        if (mode == 0 && (d.movement[i] == 1 || !d.moved[i])) continue;
        float4 q = d.rot[i];
        if (mode != 2 || d.moved[i]) {
            q = qnormalize(q);
            d.rot[i] = q;
        }
        M33 R = quatRot(q);
        f3 c = mk(d.pos[i]);
        f3 mn, mx;
        if (d.has_union && d.prim_start[i] >= 0) {
            // each primitive's AABB, the body's their combination in order
            // (ConvexUnionGeometry, RigidBody.cpp:286-294; AABB::combine)
            const int q0 = d.prim_start[i], nq = d.prim_count[i];
            for (int q = q0; q < q0 + nq; q++) {
                f3 pl, ph;
                shape_aabb(d.shapes + d.prim_shape[q], c, R, &pl, &ph);
                d.prim_lo[q] = make_float4(pl.x, pl.y, pl.z, 0.f);
                d.prim_hi[q] = make_float4(ph.x, ph.y, ph.z, 0.f);
                if (q == q0) { mn = pl; mx = ph; }
                else {
                    mn = mk(fminf(mn.x, pl.x), fminf(mn.y, pl.y), fminf(mn.z, pl.z));
                    mx = mk(fmaxf(mx.x, ph.x), fmaxf(mx.y, ph.y), fmaxf(mx.z, ph.z));
                }
            }
        } else {
            shape_aabb(d.shapes + d.shape[i], c, R, &mn, &mx);
        }
        d.aabb_lo[i] = make_float4(mn.x, mn.y, mn.z, 0.f);
        d.aabb_hi[i] = make_float4(mx.x, mx.y, mx.z, 0.f);
    }
}
}  // namespace

static int grid_for(int n, int per_block, int n_sms) {
    int g = (n + per_block - 1) / per_block;
    int cap = n_sms * 8;
    return g < 1 ? 1 : (g > cap ? cap : g);
}

void launch_gravity(const Dev& d, const Launch& L) {
    k_gravity<<<grid_for(d.n_bodies, 256, L.n_sms), 256, 0, L.st>>>(d);
}

void launch_pairs(const Dev& d, const Launch& L) {
    const int g = grid_for(d.n_bodies, 8 * kPairGroup, L.n_sms), gw = grid_for(d.n_bodies, 8, 2 * L.n_sms);
    const bool grid = d.grid_buckets > 0;
    if (grid) {
        k_grid_begin<<<17, 1024, 0, L.st>>>(d);
        k_grid_put<<<grid_for(d.n_bodies, 256, L.n_sms), 256, 0, L.st>>>(d, 0);
        k_grid_buckets<<<1, 1024, 0, L.st>>>(d);
        k_grid_put<<<grid_for(d.n_bodies, 256, L.n_sms), 256, 0, L.st>>>(d, 1);
        k_grid_count<<<gw, 256, 0, L.st>>>(d);
        k_grid_far<<<64, 1024, 0, L.st>>>(d, 0);
    }
    if (!d.all_grid) k_pairs<<<g, 256, 0, L.st>>>(d, 0);
    launch_scan<PairScan>(d, nullptr, d.n_bodies, d.n_bodies, L);
    if (grid) {
        k_grid_far<<<64, 1024, 0, L.st>>>(d, 1);
        k_grid_write<<<gw, 256, 0, L.st>>>(d);
    }
    if (!d.all_grid) k_pairs<<<g, 256, 0, L.st>>>(d, 1);
}

void launch_geometry(const Dev& d, int mode, const Launch& L) {
    k_geometry<<<grid_for(d.n_bodies, 128, L.n_sms), 128, 0, L.st>>>(d, mode);
}

}  // namespace cpgpu
