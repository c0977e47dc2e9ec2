// orbgpu_mappoint.cu -- MapPoint::ComputeDistinctiveDescriptors for many map
// points in one launch.
//
// The reference (src/MapPoint.cc:365-447) gathers the descriptors of the
// keyframes observing a map point (bad keyframes skipped), fills the N x N
// table of DescriptorDistance values, sorts every row, takes element
// (size_t)(0.5 * (N - 1)) as that descriptor's median distance to the others
// (itself included, at distance 0) and keeps the first descriptor with the
// least median.  Here the lists arrive as CSR: obs_offsets[m + 1] into
// obs_rows, each entry a row of a descriptor pool (the keyframes' descriptor
// matrices, resident in HBM), -1 for an observation of a bad keyframe.
//
// One warp takes 4 to 32 consecutive map points, a lane each for their list's
// bounds.  Lists of one or two need no distances: every median is the own 0,
// so the lane keeps its first valid observation.  The others go to lane groups
// of 4, 8, 16 or 32, the smallest that holds the list, each lane holding one
// observation's descriptor; the lists of a group's width are numbered over
// the warp's map points, so that a pass takes 8, 4, 2 or 1 of them and only
// the last is not full.  The group's descriptors sit in shared memory.  In
// groups up to 16 every lane computes the distances to the next G/2 lanes of
// its group (cyclically) and receives the other half from the lanes before it
// (distances are symmetric), then sorts its row with Batcher's odd-even
// network and reads element k.  In a group of 32 the cycle is the list's own
// length, and element k is found by binary lifting over the distance range
// 0..256 on 16-bit pairs.  The group's minimum of (median, lane) is the
// reference's first least median.
// Longer lists (more than 32 observations) run one map point per warp: rows
// in chunks of 32 lanes, each row's median from two histogram passes (d >> 4,
// then d & 15 inside the coarse bin) in lane-private shared-memory columns.
//
// Bound by issue: the distances are a tenth of the instructions, the rest is
// lanes without an observation, sorts and bookkeeping (fixed groups of 4
// map points, without the width of 4, took 261 instructions a map point).  A
// million map points of 6 observations 463 -> 285 us, of 3 187 -> 87.
#include <algorithm>

#include "orbgpu_host.h"

namespace orbgpu {

#define DD_WARPS 4          // warps per block
#define DD_BLOCKS_PER_SM 8  // resident blocks per SM (64 registers x 128 threads)

struct DDArgs {
    const uint4* pool;  // pool_rows x 32 bytes
    int pool_rows;
    const int* offsets;  // m + 1
    const int* rows;     // n_obs
    int n_obs;
    int m;
    int per_warp;  // map points a warp takes (4 to 32)
    int* best;   // m
    uint4* out;  // m x 32 bytes, or null
};

struct DDShared {
    uint4 desc[DD_WARPS][2][32];  // one warp's staged descriptors (low, high halves)
    unsigned char order[DD_WARPS][32];  // lanes of the lists of one width, in order
    int hist[DD_WARPS][17][32];   // lane-private histogram columns (long lists)
};

#define DD_FULL 0xffffffffu

// Element k of a row whose distances, the own 0 apart, are held as 16-bit
// pairs: the smallest v in 0..256 with 1 + #{d <= v} > k, by binary lifting.
// Per pair, (0x8000 + v) - d stays within its half (d <= 512, v <= 511) and
// has bit 15 set exactly when d <= v; dp2a adds the two flags.  Entries of
// absent or skipped observations hold 512 and never count; the pairs from
// 'pairs' on are all such entries.
__device__ __forceinline__ int dd_row_rank(const unsigned (&p)[16], int k, int pairs) {
    int lo = 0;
#pragma unroll 1
    for (int step = 256; step >= 1; step >>= 1) {
        const int v = lo + step - 1;
        const unsigned v2 = (unsigned)(0x8000 + v) * 0x10001u;
        unsigned acc = 0;
#pragma unroll
        for (int ic = 0; ic < 16; ic += 4) {
            if (ic >= pairs) break;
#pragma unroll
            for (int i = ic; i < ic + 4; i++) acc = __dp2a_lo((v2 - p[i]) & 0x80008000u, 0x0101u, acc);
        }
        if ((int)(acc >> 15) < k) lo += step;
    }
    return lo;
}

// Ascending sort of G registers: Batcher's odd-even merge sort (5, 19 and 63
// exchanges for 4, 8 and 16; a bitonic network has 6, 24 and 80).
template <int G, int P = 1, int K = 1>
__device__ __forceinline__ void dd_sort(int (&d)[G]) {
#pragma unroll
    for (int x = K % P; x + K < G; x++) {
        if ((x - K % P) % (2 * K) < K && x / (2 * P) == (x + K) / (2 * P)) {
            const int lo = min(d[x], d[x + K]), hi = max(d[x], d[x + K]);
            d[x] = lo;
            d[x + K] = hi;
        }
    }
    if constexpr (K > 1) dd_sort<G, P, K / 2>(d);
    else if constexpr (2 * P < G) dd_sort<G, 2 * P, 2 * P>(d);
}

__device__ __forceinline__ void dd_store(const DDArgs& a, int mp, int row, uint4 d0, uint4 d1) {
    a.best[mp] = row;
    if (a.out) {
        a.out[2 * (size_t)mp] = d0;
        a.out[2 * (size_t)mp + 1] = d1;
    }
}

// The lists of the lanes of 'mask' (all of 1..G observations from o0) in lane
// groups of width G; lane g's map point is base + g.
template <int G>
__device__ __forceinline__ void dd_group_pass(const DDArgs& a, uint4 (*sd)[32], unsigned char* order, int lane, int base,
                                              int o0_own, int n_own, unsigned mask) {
    constexpr int NG = 32 / G;
    const int grp = lane / G, l = lane % G;
    const unsigned gmask = G == 32 ? DD_FULL : ((1u << G) - 1u);
    const int count = __popc(mask);
    __syncwarp();
    if ((mask >> lane) & 1u) order[__popc(mask & ((1u << lane) - 1u))] = (unsigned char)lane;
    __syncwarp();
    for (int q = 0; q < count; q += NG) {
        const int g = q + grp < count ? order[q + grp] : -1;
        const int gs = g < 0 ? 0 : g;
        const int o0 = __shfl_sync(DD_FULL, o0_own, gs);
        const int n_of = __shfl_sync(DD_FULL, n_own, gs);
        const int n = g < 0 ? 0 : n_of;
        int r = -1;
        if (l < n) r = __ldg(a.rows + o0 + l);
        const bool valid = r >= 0 && r < a.pool_rows;
        const bool bad = l < n && (r < -1 || r >= a.pool_rows);
        const unsigned gv = (__ballot_sync(DD_FULL, valid) >> (grp * G)) & gmask;
        const bool gbad = ((__ballot_sync(DD_FULL, bad) >> (grp * G)) & gmask) != 0;
        uint4 d0 = make_uint4(0, 0, 0, 0), d1 = d0;
        if (valid) {
            d0 = __ldg(a.pool + 2 * (size_t)r);
            d1 = __ldg(a.pool + 2 * (size_t)r + 1);
        }
        __syncwarp();
        sd[0][lane] = d0;
        sd[1][lane] = d1;
        __syncwarp();
        const int nv = __popc(gv);
        const int k = (nv - 1) >> 1;
        int median;
        if constexpr (G < 32) {
            // d(l, l + s) for s = 1..G/2 here, d(l, l - s) from lane l - s
            int h[G / 2];
#pragma unroll
            for (int s = 1; s <= G / 2; s++) {
                const int j = grp * G + ((l + s) & (G - 1));
                h[s - 1] = hamming256(d0, d1, sd[0][j], sd[1][j]);
            }
            int d[G];
            d[0] = 0;
#pragma unroll
            for (int s = 1; s <= G / 2; s++) d[s] = (gv >> ((l + s) & (G - 1))) & 1u ? h[s - 1] : 512;
#pragma unroll
            for (int s = 1; s < G / 2; s++) {
                const int v = __shfl_sync(DD_FULL, h[s - 1], (l - s) & (G - 1), G);
                d[G / 2 + s] = (gv >> ((l - s) & (G - 1))) & 1u ? v : 512;
            }
            dd_sort<G>(d);
            median = d[0];
#pragma unroll
            for (int i = 1; i < G / 2; i++) median = i == k ? d[i] : median;
        } else {
            // step t + 1: the distances to the lanes t + 1 after and before, cyclically over the list
            const int pairs = n >> 1;
            unsigned p[16];
#pragma unroll
            for (int tc = 0; tc < 16; tc += 4) {
#pragma unroll
                for (int t = tc; t < tc + 4; t++) p[t] = 512u * 0x10001u;
                if (tc < pairs) {
#pragma unroll
                    for (int t = tc; t < tc + 4; t++) {
                        const int up = l + t + 1 - (l + t + 1 >= n ? n : 0), down = l - t - 1 + (l - t - 1 < 0 ? n : 0);
                        const int h = hamming256(d0, d1, sd[0][up & 31], sd[1][up & 31]);
                        const int hd = __shfl_sync(DD_FULL, h, down & 31);
                        const bool in = 2 * (t + 1) <= n;  // at 2 (t + 1) = n both are the same lane
                        const unsigned e0 = in && ((gv >> (up & 31)) & 1u) ? (unsigned)h : 512u;
                        const unsigned e1 = in && 2 * (t + 1) < n && ((gv >> (down & 31)) & 1u) ? (unsigned)hd : 512u;
                        p[t] = e0 | (e1 << 16);
                    }
                }
            }
            median = dd_row_rank(p, k, pairs);
        }
        int key = valid ? (median << 5) | l : 0x7fffffff;
#pragma unroll
        for (int s = G / 2; s >= 1; s >>= 1) key = min(key, __shfl_xor_sync(DD_FULL, key, s));
        if (g >= 0) {
            const int mp = base + g;
            if (gbad) {
                if (l == 0) a.best[mp] = -2;
            } else if (nv == 0) {
                if (l == 0) a.best[mp] = -1;
            } else if (l == (key & 31)) {
                dd_store(a, mp, r, d0, d1);
            }
        }
    }
}

// One map point with more than 32 observations, the whole warp.
__device__ __forceinline__ void dd_long_list(const DDArgs& a, uint4 (*sd)[32], int (*hist)[32], int lane, int mp, int o0, int n) {
    int nv = 0;
    bool bad = false;
    for (int c = 0; c < n; c += 32) {
        const bool in = c + lane < n;
        const int r = in ? __ldg(a.rows + o0 + c + lane) : -1;
        nv += __popc(__ballot_sync(DD_FULL, r >= 0 && r < a.pool_rows));
        bad |= __ballot_sync(DD_FULL, in && (r < -1 || r >= a.pool_rows)) != 0;
    }
    if (bad || nv == 0) {
        if (lane == 0) a.best[mp] = bad ? -2 : -1;
        return;
    }
    const int k = (nv - 1) >> 1;
    const uint4 z = make_uint4(0, 0, 0, 0);
    unsigned long long best = ~0ull;
    for (int rc = 0; rc < n; rc += 32) {
        const int i = rc + lane;
        const int ri = i < n ? __ldg(a.rows + o0 + i) : -1;
        const bool vi = ri >= 0;
        uint4 m0 = z, m1 = z;
        if (vi) {
            m0 = __ldg(a.pool + 2 * (size_t)ri);
            m1 = __ldg(a.pool + 2 * (size_t)ri + 1);
        }
        int coarse = 0, below = 0, median = 0;
        for (int pass = 0; pass < 2; pass++) {
#pragma unroll
            for (int b = 0; b < 17; b++) hist[b][lane] = 0;
            for (int jc = 0; jc < n; jc += 32) {
                const int rj = jc + lane < n ? __ldg(a.rows + o0 + jc + lane) : -1;
                const unsigned vj = __ballot_sync(DD_FULL, rj >= 0);
                uint4 b0 = z, b1 = z;
                if (rj >= 0) {
                    b0 = __ldg(a.pool + 2 * (size_t)rj);
                    b1 = __ldg(a.pool + 2 * (size_t)rj + 1);
                }
                __syncwarp();
                sd[0][lane] = b0;
                sd[1][lane] = b1;
                __syncwarp();
                if (vi) {
                    const int jn = min(32, n - jc);
#pragma unroll 2
                    for (int jj = 0; jj < jn; jj++) {
                        if (!((vj >> jj) & 1u)) continue;
                        const int d = hamming256(m0, m1, sd[0][jj], sd[1][jj]);
                        // an atomic without a result: the next distance does not wait for the count
                        if (pass == 0) atomicAdd(&hist[d >> 4][lane], 1);
                        else if ((d >> 4) == coarse) atomicAdd(&hist[d & 15][lane], 1);
                    }
                }
            }
            if (vi) {
                // element k lies in the first bin where the running count passes k
                int cum = pass == 0 ? 0 : below;
                const int nb = pass == 0 ? 17 : 16;
                for (int b = 0; b < nb; b++) {
                    const int c = hist[b][lane];
                    if (cum + c > k) {
                        if (pass == 0) {
                            coarse = b;
                            below = cum;
                        } else {
                            median = coarse * 16 + b;
                        }
                        break;
                    }
                    cum += c;
                }
            }
        }
        if (vi) {
            const unsigned long long key = ((unsigned long long)median << 32) | (unsigned)i;
            best = key < best ? key : best;
        }
    }
    best = warp_min_u64(best);
    if (lane == 0) {
        const int r = __ldg(a.rows + o0 + (int)(best & 0xffffffffu));
        dd_store(a, mp, r, __ldg(a.pool + 2 * (size_t)r), __ldg(a.pool + 2 * (size_t)r + 1));
    }
}

__global__ void __launch_bounds__(DD_WARPS * 32, DD_BLOCKS_PER_SM) k_distinctive_descriptors(const __grid_constant__ DDArgs a) {
    __shared__ DDShared sh;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned at = (blockIdx.x * DD_WARPS + w) * (unsigned)a.per_warp;
    if (at >= (unsigned)a.m) return;
    const int base = (int)at;
    const bool mine = lane < a.per_warp && lane < a.m - base;
    int o0 = 0, n = 0;
    if (mine) {
        o0 = __ldg(a.offsets + base + lane);
        const int o1 = __ldg(a.offsets + base + lane + 1);
        n = o1 - o0;
        if (o0 < 0 || n < 0 || o1 > a.n_obs) {
            a.best[base + lane] = -2;
            n = 0;
        } else if (n <= 2) {
            const int r0 = n > 0 ? __ldg(a.rows + o0) : -1, r1 = n > 1 ? __ldg(a.rows + o0 + 1) : -1;
            const int r = r0 >= 0 ? r0 : r1;
            if (r0 < -1 || r0 >= a.pool_rows || r1 < -1 || r1 >= a.pool_rows) a.best[base + lane] = -2;
            else if (r < 0) a.best[base + lane] = -1;
            else dd_store(a, base + lane, r, __ldg(a.pool + 2 * (size_t)r), __ldg(a.pool + 2 * (size_t)r + 1));
        }
    }
    __syncwarp();
    const unsigned c4 = __ballot_sync(DD_FULL, n > 2 && n <= 4), c8 = __ballot_sync(DD_FULL, n > 4 && n <= 8);
    const unsigned c16 = __ballot_sync(DD_FULL, n > 8 && n <= 16), c32 = __ballot_sync(DD_FULL, n > 16 && n <= 32);
    unsigned clong = __ballot_sync(DD_FULL, n > 32);
    if (c4) dd_group_pass<4>(a, sh.desc[w], sh.order[w], lane, base, o0, n, c4);
    if (c8) dd_group_pass<8>(a, sh.desc[w], sh.order[w], lane, base, o0, n, c8);
    if (c16) dd_group_pass<16>(a, sh.desc[w], sh.order[w], lane, base, o0, n, c16);
    if (c32) dd_group_pass<32>(a, sh.desc[w], sh.order[w], lane, base, o0, n, c32);
    while (clong) {
        const int g = __ffs(clong) - 1;
        clong &= clong - 1;
        const int of = __shfl_sync(DD_FULL, o0, g), nf = __shfl_sync(DD_FULL, n, g);
        dd_long_list(a, sh.desc[w], sh.hist[w], lane, base + g, of, nf);
    }
}

}  // namespace orbgpu

using namespace orbgpu;

extern "C" int orbgpu_distinctive_descriptors(const uint8_t* pool, int pool_rows, const int* obs_offsets,
                                              const int* obs_rows, int n_obs, int m, int* best_rows,
                                              uint8_t* descriptors, void* stream) {
    if (m < 0 || pool_rows < 0 || n_obs < 0 || (m > 0 && (!obs_offsets || !best_rows)) ||
        (pool_rows > 0 && !pool) || (n_obs > 0 && !obs_rows)) {
        orbgpu_set_last_error("orbgpu_distinctive_descriptors: negative size or missing array", __FILE__, __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    if (((uintptr_t)pool & 15) || ((uintptr_t)descriptors & 15)) {
        orbgpu_set_last_error("orbgpu_distinctive_descriptors: pool and descriptors must be 16-byte aligned", __FILE__,
                              __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    if (m == 0) return ORBGPU_OK;
    DDArgs a;
    a.pool = reinterpret_cast<const uint4*>(pool);
    a.pool_rows = pool_rows;
    a.offsets = obs_offsets;
    a.rows = obs_rows;
    a.n_obs = n_obs;
    a.m = m;
    a.best = best_rows;
    a.out = reinterpret_cast<uint4*>(descriptors);
    // a block takes its map points once and ends, so that the device evens out
    // long and short lists (a million map points in rounds over resident
    // blocks: 346 us against 285); as many per warp (fuller groups) as leave
    // every resident warp some
    const long long warps = (long long)nsm_of_current_device() * DD_BLOCKS_PER_SM * DD_WARPS;
    a.per_warp = (int)std::min(32LL, std::max(4LL, (m + warps - 1) / warps));
    const int per_block = DD_WARPS * a.per_warp, blocks = (int)(((long long)m + per_block - 1) / per_block);
    k_distinctive_descriptors<<<blocks, DD_WARPS * 32, 0, (cudaStream_t)stream>>>(a);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    return ORBGPU_OK;
}
