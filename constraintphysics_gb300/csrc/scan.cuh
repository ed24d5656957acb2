// scan.cuh — exclusive prefix of device-counted values in one launch.
//
// A step needs five of them, each between two kernels that read and write the
// same items, and most are short: what they cost is launches.  One kernel
// computes the values (Op::in(d, i)), their prefix (Op::out(d, i, prefix)) and
// what follows from the total (Op::done(d, total), one thread), where separate kernels for the
// values, chunk sums, their prefix, its addition and the total's check took
// five launches of 2-3 us each.
//
// The decoupled look-back prefix of Merrill and Garland ("Single-pass Parallel
// Prefix Scan with Decoupled Look-back", 2016).  Chunks are taken in order from
// a counter.  A chunk's block publishes its sum, then finds the sum of the
// chunks before it by looking back at theirs, 32 at a time (sums, or a prefix
// where one is known).  A block only ever waits for chunks that other blocks
// have already taken, so it makes progress whatever else runs; the wait is
// bounded like every other (ST_TIMEOUT).
#pragma once
#include <algorithm>

#include "kernels.cuh"

namespace cpgpu {

constexpr int kScanWaitLimit = 1 << 20;   // polls before a chunk gives up on its predecessors
constexpr int kScanThreads = 512, kScanPer = 4, kScanChunk = kScanThreads * kScanPer;

// a chunk's published word: bits 0-31 value, 32-33 state (1 its sum, 2 the
// prefix up to and including it), 34- the launch it belongs to
__device__ __forceinline__ unsigned long long scan_word(unsigned epoch, unsigned state, int v) {
    return ((unsigned long long)epoch << 34) | ((unsigned long long)state << 32) | (unsigned)v;
}

template <class Op>
__global__ void __launch_bounds__(kScanThreads) k_scan(Dev d, const int* n_dev, int n_host) {
    ScanTmp* tmp = d.scan_tmp;
    __shared__ int ws[kScanThreads / 32], sh_chunk, sh_before, sh_last;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int n = n_dev ? *n_dev : n_host;
    const int chunks = max(1, (n + kScanChunk - 1) / kScanChunk);
    const unsigned epoch = *(volatile unsigned*)&tmp->epoch & 0x3fffffffu;
    while (true) {
        __syncthreads();   // the previous chunk's shared values are no longer read
        if (tid == 0) sh_chunk = atomicAdd(&tmp->next, 1);
        __syncthreads();
        const int c = sh_chunk;
        if (c >= chunks) break;
        const int i0 = c * kScanChunk + tid * kScanPer;
        int v[kScanPer], sum = 0;
#pragma unroll
        for (int k = 0; k < kScanPer; k++) {
            v[k] = i0 + k < n ? Op::in(d, i0 + k) : 0;
            sum += v[k];
        }
        int x = sum;
        for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += t; }
        if (lane == 31) ws[wid] = x;
        __syncthreads();
        if (wid == 0) {
            int y = lane < kScanThreads / 32 ? ws[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, y, o); if (lane >= o) y += t; }
            const int total = __shfl_sync(0xffffffffu, y, 31);
            if (lane < kScanThreads / 32) ws[lane] = y;
            volatile unsigned long long* word = tmp->word;
            if (lane == 0) word[c] = scan_word(epoch, c == 0 ? 2 : 1, total);
            int before = 0;
            long long polls = 0;
            for (int p = c - 1; p >= 0;) {   // chunks p, p - 1, ..., p - 31
                const int q = p - lane;
                const unsigned long long w = q >= 0 ? word[q] : scan_word(epoch, 2, 0);
                const bool ready = (unsigned)(w >> 34) == epoch && ((w >> 32) & 3) != 0;
                const unsigned pre = __ballot_sync(0xffffffffu, ready && ((w >> 32) & 3) == 2);
                const int last = pre ? __ffs(pre) - 1 : 31;   // lanes 0 .. last are needed
                if (!__all_sync(0xffffffffu, ready || lane > last)) {
                    if (++polls < kScanWaitLimit) continue;
                    if (lane == 0) atomicOr(d.status, ST_TIMEOUT);
                    break;
                }
                before += __reduce_add_sync(0xffffffffu, lane <= last ? (int)(unsigned)w : 0);
                if (pre) break;
                p -= 32;
            }
            if (lane == 0) {
                if (c > 0) word[c] = scan_word(epoch, 2, before + total);
                sh_before = before;
                if (c == chunks - 1) Op::done(d, before + total);
            }
        }
        __syncthreads();
        int run = sh_before + x - sum + (wid > 0 ? ws[wid - 1] : 0);
#pragma unroll
        for (int k = 0; k < kScanPer; k++) {
            if (i0 + k < n) Op::out(d, i0 + k, run);
            run += v[k];
        }
    }
    // the last block to leave readies the counters for the next launch
    if (tid == 0) sh_last = atomicAdd(&tmp->left, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (sh_last && tid == 0) {
        tmp->next = 0;
        tmp->left = 0;
        *(volatile unsigned*)&tmp->epoch = epoch + 1;
    }
}

// `cap`: bound on the item count (n_host, or *n_dev when n_dev is not null)
template <class Op>
void launch_scan(const Dev& d, const int* n_dev, int n_host, int cap, const Launch& L) {
    const int grid = std::max(1, std::min((cap + kScanChunk - 1) / kScanChunk, L.n_sms));
    k_scan<Op><<<grid, kScanThreads, 0, L.st>>>(d, n_dev, n_host);
}

}  // namespace cpgpu
