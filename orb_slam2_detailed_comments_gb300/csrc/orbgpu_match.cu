// orbgpu_match.cu -- the windowed descriptor searches and stereo matching.
//
// Distances and candidate windows are computed in parallel (one warp per
// query, or half of one); the parts of the reference that are sequential by
// construction -- a later query seeing the matches of earlier ones
// (vMatchedDistance in SearchForInitialization, claimed keypoints in
// SearchByProjection) -- are resolved as fixed points over the precomputed
// candidate lists.
//
// Candidate order: Frame::GetFeaturesInArea (src/Frame.cc:590-670) visits
// grid cells column by column and each cell in keypoint-index order, so a
// candidate's position in that order is (cell x * 48 + cell y, index).  The
// searches compare candidates lexicographically on (distance, position),
// which reproduces the reference's "first strictly smaller wins" loops.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "orbgpu_grid.cuh"
#include "orbgpu_host.h"
#include "orbgpu_stereo.cuh"

namespace orbgpu {

#define PROJ_ROUNDS 12
#define PROJ_NONE 0x7f7f7f7f

struct GridDev {
    const orbgpu_keypoint* kps;
    const uint8_t* desc;
    const float* uright;
    int n;
    float minX, minY, invW, invH;
    const int* cell_start;  // 64*48 + 1
    const GridRec* recs;    // n
    float scale[16];
};

// A frame's grid: one block up to GRID_BLOCK_N keypoints (one launch, in
// shared memory), three launches over global counters beyond.
#define GRID_BLOCK_N 8192
__global__ void __launch_bounds__(1024) k_grid_build(const orbgpu_keypoint* kps, int n, float minX, float minY, float invW,
                                                     float invH, int* cell_start, GridRec* recs) {
    grid_build_block(kps, n, minX, minY, invW, invH, cell_start, recs);
}

__global__ void k_grid_count(const orbgpu_keypoint* kps, int n, float minX, float minY, float invW, float invH,
                             int* cell_count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = pos_in_grid(kps[i], minX, minY, invW, invH);
    if (c >= 0) atomicAdd(&cell_count[c], 1);
}

__global__ void k_grid_scan(const int* cell_count, int* cell_start, int* cursor) {
    __shared__ int s_scan[32];
    const int ncell = ORBGPU_GRID_CELLS;
    int base = 0;
    for (int b0 = 0; b0 < ncell; b0 += blockDim.x) {
        const int c = b0 + threadIdx.x;
        const int v = c < ncell ? cell_count[c] : 0;
        int tot;
        const int ex = block_exclusive_scan(v, s_scan, &tot);
        if (c < ncell) {
            cell_start[c] = base + ex;
            cursor[c] = base + ex;
        }
        base += tot;
    }
    if (threadIdx.x == 0) cell_start[ncell] = base;
}

__global__ void k_grid_fill(const orbgpu_keypoint* kps, int n, float minX, float minY, float invW, float invH, int* cursor,
                            GridRec* recs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const orbgpu_keypoint kp = kps[i];
    const int c = pos_in_grid(kp, minX, minY, invW, invH);
    if (c >= 0) recs[atomicAdd(&cursor[c], 1)] = grid_rec(kp, c, i);
}

// Frame::GetFeaturesInArea cell range; false when the window misses the grid.
__device__ __forceinline__ bool area_cells(const GridDev& g, float x, float y, float r, int& x0, int& x1, int& y0,
                                           int& y1) {
    x0 = max(0, (int)floorf(__fmul_rn(__fsub_rn(__fsub_rn(x, g.minX), r), g.invW)));
    if (x0 >= ORBGPU_GRID_COLS) return false;
    x1 = min(ORBGPU_GRID_COLS - 1, (int)ceilf(__fmul_rn(__fadd_rn(__fsub_rn(x, g.minX), r), g.invW)));
    if (x1 < 0) return false;
    y0 = max(0, (int)floorf(__fmul_rn(__fsub_rn(__fsub_rn(y, g.minY), r), g.invH)));
    if (y0 >= ORBGPU_GRID_ROWS) return false;
    y1 = min(ORBGPU_GRID_ROWS - 1, (int)ceilf(__fmul_rn(__fadd_rn(__fsub_rn(y, g.minY), r), g.invH)));
    if (y1 < 0) return false;
    return true;
}

__device__ __forceinline__ bool in_area(const GridRec& rec, float x, float y, float r, int minLevel, int maxLevel) {
    const bool check = (minLevel > 0) || (maxLevel >= 0);
    if (check) {
        if (rec.octave() < minLevel) return false;
        if (maxLevel >= 0 && rec.octave() > maxLevel) return false;
    }
    return in_disc(rec, x, y, __fmul_rn(r, r));
}

// The records of the grid cells [x0, x1] x [y0, y1] for one whole warp.
template <typename Visit>
__device__ __forceinline__ void warp_window_recs(const GridDev& g, int x0, int x1, int y0, int y1, Visit visit) {
    seg_window_recs<32>(g.cell_start, g.recs, true, x0, x1, y0, y1, visit);
}

__device__ __forceinline__ uint64_t cand_key(int dist, int cell, int idx) {
    return ((uint64_t)(uint32_t)dist << 40) | ((uint64_t)(uint32_t)cell << 20) | (uint64_t)(uint32_t)idx;
}

// A query's row of candidate keys: of slot_cap keys from slots on, one row
// after the other, or from slots[start[i]] on where start is given (64-bit keys
// only: rows of the queries' own lengths).
template <typename Key>
__device__ __forceinline__ Key* cand_row(Key* slots, int slot_cap, const long long* start, int i) {
    if constexpr (sizeof(Key) > sizeof(uint32_t))
        if (start) return slots + start[i];
    return slots + (size_t)i * slot_cap;
}

// ----------------------------------------------------------------- SearchForInitialization
// The candidates of every level-0 keypoint of F1 in the window around
// prev[i1] (src/ORBmatcher.cc:603-640), one warp each, into rows of slot_cap
// keys.  A candidate with nnratio * dist > TH_LOW (nnratio <= 1) can neither be
// accepted (dist > TH_LOW) nor make an accepted best fail the ratio test (best
// <= TH_LOW < nnratio * dist): the lists leave it out, and with it all but a
// few of a window's keypoints.
__global__ void k_init_candidates(GridDev g2, const orbgpu_keypoint* kps1, const uint8_t* desc1, int n1,
                                  const float* prev, float window, float nnratio, int slot_cap, const long long* start,
                                  uint64_t* slots, int* slot_count, int* status) {
    const bool drop_far = nnratio <= 1.0f;
    const int lane = threadIdx.x & 31;
    const int i1 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i1 >= n1) return;
    const int octave = kps1[i1].octave;
    int total = 0;
    int x0, x1, y0, y1;
    if (octave <= 0 && area_cells(g2, prev[2 * i1], prev[2 * i1 + 1], window, x0, x1, y0, y1)) {
        const uint4* d1 = reinterpret_cast<const uint4*>(desc1 + (size_t)i1 * 32);
        const uint4 a0 = d1[0], a1 = d1[1];
        const float px = prev[2 * i1], py = prev[2 * i1 + 1];
        uint64_t* row = cand_row(slots, slot_cap, start, i1);
        warp_window_recs(g2, x0, x1, y0, y1, [&](const GridRec& rec, bool valid) {
            bool ok = valid && in_area(rec, px, py, window, octave, octave);
            int dist = 256;
            if (ok) {
                const uint4* d2 = reinterpret_cast<const uint4*>(g2.desc + (size_t)rec.idx * 32);
                dist = hamming256(a0, a1, d2[0], d2[1]);
                ok = !(drop_far && __fmul_rn((float)dist, nnratio) > (float)ORBGPU_TH_LOW);
            }
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            const int pos = total + __popc(m & ((1u << lane) - 1));
            if (ok && pos < slot_cap) row[pos] = cand_key(dist, rec.cell(), (int)rec.idx);
            total += __popc(m);
        });
    }
    if (lane == 0) {
        slot_count[i1] = total;
        if (total > slot_cap) atomicMax(status, total);
    }
}

__global__ void k_exclusive_scan(const int* in, int n, int* out, int* total) {
    __shared__ int s_scan[32];
    int base = 0;
    for (int b0 = 0; b0 < n; b0 += blockDim.x) {
        const int i = b0 + threadIdx.x;
        const int v = i < n ? in[i] : 0;
        int tot;
        const int ex = block_exclusive_scan(v, s_scan, &tot);
        if (i < n) out[i] = base + ex;
        base += tot;
    }
    if (threadIdx.x == 0) *total = base;
}

// The in-order resolution of src/ORBmatcher.cc:600-677 by one block, as a
// fixed point.  In the reference keypoint i of F1 skips candidate j when an
// earlier keypoint took j at a distance not above its own (vMatchedDistance
// holds the last taker's, which is also the least), takes its best remaining
// candidate if that passes TH_LOW and the ratio test, and a later taker of j
// ends the earlier one's match.  Round r evaluates every keypoint against the
// choices of round r - 1, kept as one list of takers per F2 keypoint; once a
// round changes no choice, the choices are the sequential ones (by induction
// over the keypoints: round r fixes the first r + 1).  The match of an F2
// keypoint is then its last taker's, and the rotation histogram counts every
// taker.  A warp walking the keypoints in order took 236 us at 640 x 480 /
// 1000 features, this 9.  Keypoints that depend on one another in a long chain
// (a row of alike features, each with a second candidate that the one before
// leaves it) settle one a round: after INIT_ROUNDS rounds, or where a list of
// takers passes INIT_TAKERS, the warp's walk decides after all, so that the
// time stays linear in the keypoints.  Arrays (shared memory when 'local', else
// global): choice and its distance (n1 each), two sets of list heads (n2) and
// links (n1).
#define INIT_ROUNDS 64
#define INIT_TAKERS 4096
// (best, second): the least (distance, position) key and the least distance of
// the others, with one more key.
__device__ __forceinline__ void init_insert(uint64_t key, uint64_t& best, int& second) {
    const uint64_t other = key < best ? best : key;
    best = key < best ? key : best;
    if (other != ~0ull) second = min(second, (int)(other >> 40));
}
__device__ __forceinline__ bool init_accepts(uint64_t best, int second, float nnratio) {
    const int d = (int)(best >> 40);
    return best != ~0ull && d <= ORBGPU_TH_LOW && (float)d < __fmul_rn((float)second, nnratio);
}
// The walk, by the calling warp: choice[n1]; least[n2] (the matched distances)
// holds 0x7fffffff before.
__device__ __forceinline__ void init_walk(int n1, int slot_cap, const long long* start, const int* slot_count,
                                          const uint64_t* slots, float nnratio, int* choice, int* least) {
    const int lane = threadIdx.x & 31;
    for (int i0 = 0; i0 < n1; i0 += 32) {
        const int mine = i0 + lane < n1 ? min(slot_count[i0 + lane], slot_cap) : 0;
        if (i0 + lane < n1) choice[i0 + lane] = -1;
        __syncwarp();
        unsigned todo = __ballot_sync(0xffffffffu, mine > 0);
        while (todo) {
            const int t = __ffs(todo) - 1, cnt = __shfl_sync(0xffffffffu, mine, t);
            todo &= todo - 1;
            const uint64_t* row = cand_row(slots, slot_cap, start, i0 + t);
            uint64_t best = ~0ull;
            int second = 0x7fffffff;
            for (int e = lane; e < cnt; e += 32) {
                const uint64_t key = row[e];
                if (least[key & 0xFFFFF] > (int)(key >> 40)) init_insert(key, best, second);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const uint64_t ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int os = __shfl_xor_sync(0xffffffffu, second, o);
                second = min(second, os);
                init_insert(ob, best, second);
            }
            if (lane == 0 && init_accepts(best, second, nnratio)) {
                choice[i0 + t] = (int)(best & 0xFFFFF);
                least[best & 0xFFFFF] = (int)(best >> 40);
            }
            __syncwarp();  // lane 0's update is seen by the next keypoint's filter
        }
    }
}
__host__ __device__ inline size_t init_resolve_bytes(int n1, int n2) { return 4 * (4 * (size_t)n1 + 2 * (size_t)n2); }
__global__ void __launch_bounds__(1024, 1)
    k_init_resolve(const orbgpu_keypoint* kps1, int n1, const orbgpu_keypoint* kps2, int n2, int slot_cap,
                   const long long* start, const int* slot_count, const uint64_t* slots, float nnratio, int check_ori,
                   int local, int* work, int* matches12, int* nmatches_out) {
    extern __shared__ int s_init[];
    __shared__ int hist[ORBGPU_HISTO_LENGTH];
    __shared__ int s_flag[3], s_long, s_nm, s_ind[3];
    const int tid = threadIdx.x, nt = blockDim.x;
    int* const choice = local ? s_init : work;  // n1: F2 keypoint or -1
    int* const cdist = choice + n1;             // n1
    int *head_r = cdist + n1, *head_w = head_r + n2, *next_r = head_w + n2, *next_w = next_r + n1;
    if (tid < ORBGPU_HISTO_LENGTH) hist[tid] = 0;
    if (tid < 3) s_flag[tid] = 0;
    if (tid == 0) s_nm = s_long = 0;
    for (int j = tid; j < n2; j += nt) head_r[j] = head_w[j] = -1;
    for (int i = tid; i < n1; i += nt) choice[i] = -2;
    bool converged = false;
    for (int round = 0; round < INIT_ROUNDS && !converged; round++) {
        if (tid == 0) s_flag[(round + 1) % 3] = 0;
        __syncthreads();
        // the choices' distances of the round before are read below, this
        // round's are written after the barrier
        int mine[2], mdist[2], q = 0;
        auto eval = [&](int i, int& r, int& rd) {
            const int cnt = min(slot_count[i], slot_cap);
            const uint64_t* row = cand_row(slots, slot_cap, start, i);
            uint64_t best = ~0ull;
            int second = 0x7fffffff;
            for (int e = 0; e < cnt; e++) {
                const uint64_t key = row[e];
                const int dist = (int)(key >> 40), j = (int)(key & 0xFFFFF);
                bool taken = false;
                int k = head_r[j], seen = 0;
                for (; k >= 0 && !taken && seen < INIT_TAKERS; k = next_r[k], seen++) taken = k < i && cdist[k] <= dist;
                if (taken) continue;
                if (k >= 0) s_long = 1;
                init_insert(key, best, second);
            }
            r = init_accepts(best, second, nnratio) ? (int)(best & 0xFFFFF) : -1;
            rd = (int)(best >> 40);
        };
        const bool few = n1 <= 2 * nt;  // results wait in registers, else in the links' spare array
        for (int i = tid; i < n1; i += nt, q++) {
            int r, rd;
            eval(i, r, rd);
            if (few) {
                mine[q & 1] = r;
                mdist[q & 1] = rd;
            } else {
                next_w[i] = r < 0 ? -1 : (int)(((uint32_t)rd << 20) | (uint32_t)r);  // dist <= 50, index below 2^20
            }
        }
        __syncthreads();
        q = 0;
        for (int i = tid; i < n1; i += nt, q++) {
            int r, rd;
            if (few) {
                r = mine[q & 1];
                rd = mdist[q & 1];
            } else {
                const int v = next_w[i];
                r = v < 0 ? -1 : v & 0xFFFFF;
                rd = v >> 20;
            }
            if (r != choice[i]) {
                choice[i] = r;
                s_flag[round % 3] = 1;
            }
            cdist[i] = rd;
            if (r >= 0) next_w[i] = atomicExch(&head_w[r], i);
        }
        __syncthreads();
        if (s_long) break;
        converged = s_flag[round % 3] == 0;
        int* t = head_r;
        head_r = head_w;
        head_w = t;
        t = next_r;
        next_r = next_w;
        next_w = t;
        if (!converged)
            for (int j = tid; j < n2; j += nt) head_w[j] = -1;
    }
    int* const owner = head_w;
    __syncthreads();
    if (!converged) {
        for (int j = tid; j < n2; j += nt) owner[j] = 0x7fffffff;
        __syncthreads();
        if (tid < 32) init_walk(n1, slot_cap, start, slot_count, slots, nnratio, choice, owner);
        __syncthreads();
    }
    // the owner of each F2 keypoint: its last taker
    for (int j = tid; j < n2; j += nt) owner[j] = -1;
    __syncthreads();
    const float factor = __fdiv_rn((float)ORBGPU_HISTO_LENGTH, 360.0f);
    int* const bin_of = next_w;
    for (int i = tid; i < n1; i += nt) {
        const int j = choice[i];
        int bin = -1;
        if (j >= 0) {
            atomicMax(&owner[j], i);
            if (check_ori) {
                float rot = __fsub_rn(kps1[i].angle, kps2[j].angle);
                if (rot < 0.0f) rot = __fadd_rn(rot, 360.0f);
                bin = (int)roundf(__fmul_rn(rot, factor));
                if (bin == ORBGPU_HISTO_LENGTH) bin = 0;
                atomicAdd(&hist[bin], 1);
            }
        }
        bin_of[i] = bin;
    }
    __syncthreads();
    if (tid == 0) {
        int ind1 = -1, ind2 = -1, ind3 = -1;
        int max1 = 0, max2 = 0, max3 = 0;
        for (int i = 0; i < ORBGPU_HISTO_LENGTH; i++) {  // ComputeThreeMaxima, src/ORBmatcher.cc:2035-2077
            const int sz = hist[i];
            if (sz > max1) {
                max3 = max2; max2 = max1; max1 = sz;
                ind3 = ind2; ind2 = ind1; ind1 = i;
            } else if (sz > max2) {
                max3 = max2; max2 = sz;
                ind3 = ind2; ind2 = i;
            } else if (sz > max3) {
                max3 = sz;
                ind3 = i;
            }
        }
        if ((float)max2 < __fmul_rn(0.1f, (float)max1)) {
            ind2 = -1;
            ind3 = -1;
        } else if ((float)max3 < __fmul_rn(0.1f, (float)max1)) {
            ind3 = -1;
        }
        s_ind[0] = ind1;
        s_ind[1] = ind2;
        s_ind[2] = ind3;
    }
    __syncthreads();
    int nm = 0;
    for (int i = tid; i < n1; i += nt) {
        const int j = choice[i], b = bin_of[i];
        const bool kept = j >= 0 && owner[j] == i && (b < 0 || b == s_ind[0] || b == s_ind[1] || b == s_ind[2]);
        matches12[i] = kept ? j : -1;
        nm += kept;
    }
    nm = warp_sum(nm);
    if ((tid & 31) == 0 && nm) atomicAdd(&s_nm, nm);
    __syncthreads();
    if (tid == 0) *nmatches_out = s_nm;
}

// ----------------------------------------------------------------- SearchByProjection(Frame, MapPoints)
// The candidate rows (proj_candidates: 16 lanes per map point).
#define PROJ_SEG 16
template <typename Key>
__global__ void k_proj_candidates(GridDev g, const orbgpu_mappoint* mps, const uint8_t* mp_desc, int m, float th,
                                  float nnratio, int slot_cap, const long long* start, Key* slots, int* slot_count,
                                  int* status) {
    const int lane = threadIdx.x & 31;
    const int imp = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 / PROJ_SEG) + lane / PROJ_SEG;
    const bool have = imp < m;
    if (__all_sync(0xffffffffu, !have)) return;
    orbgpu_mappoint mp{};
    if (have) mp = mps[imp];
    const ProjFrame F{g.cell_start, g.recs, g.desc, g.uright, g.minX, g.minY, g.invW, g.invH, g.scale};
    const int total = proj_candidates<PROJ_SEG, Key>(F, mp, have, mp_desc + (size_t)imp * 32, th, nnratio,
                                                     cand_row(slots, slot_cap, have ? start : nullptr, imp), slot_cap);
    if (have && (lane & (PROJ_SEG - 1)) == 0) {
        slot_count[imp] = total;
        if (total > slot_cap) atomicMax(status, total);
    }
}

// The resolution in one block (proj_resolve_block); status[1] set if it did
// not converge.
__global__ void __launch_bounds__(1024) k_proj_resolve_smem(const orbgpu_keypoint* kps, int n, int m, const uint32_t* slots,
                                                            int slot_cap, const int* slot_count, float nnratio,
                                                            const uint8_t* claimed, int* match_out, int* nmatches,
                                                            int* status) {
    extern __shared__ __align__(16) int s_dyn[];
    const int rounds = proj_resolve_block(kps, n, m, slots, slot_cap, slot_count, nullptr, nnratio, claimed, s_dyn, match_out,
                                          nmatches);
    if (threadIdx.x == 0 && rounds == 0) status[1] = 1;
}

// The same for frames that do not fit in shared memory: fixed-point rounds in
// global memory, one launch each, and a serial replay if none converged.
// In-order resolution (src/ORBmatcher.cc:117-180) by one warp.
// claimed[] starts with the caller's pre-claimed keypoints.
__global__ void k_proj_resolve(GridDev g, int m, int slot_cap, const long long* start, const int* slot_count,
                               const uint64_t* slots, float nnratio, int* match_out, int* nmatches_out, const int* converged_flags) {
    if (converged_flags && converged_flags[PROJ_ROUNDS - 1] == 0) return;
    const int lane = threadIdx.x;
    int nmatches = 0;
    for (int imp = 0; imp < m; imp++) {
        const int cnt = min(slot_count[imp], slot_cap);
        const uint64_t* row = cand_row(slots, slot_cap, start, imp);
        if (cnt == 0) continue;
        uint64_t best = ~0ull, second = ~0ull;
        for (int b = 0; b < cnt; b += 32) {
            uint64_t key = ~0ull;
            if (b + lane < cnt) {
                key = row[b + lane];
                const int idx = (int)(key & 0xFFFFF);
                if (match_out[idx] != -1 || (int)(key >> 40) >= 256) key = ~0ull;
            }
            if (key < best) {
                second = best;
                best = key;
            } else if (key < second) {
                second = key;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const uint64_t ob = __shfl_xor_sync(0xffffffffu, best, o);
            const uint64_t os = __shfl_xor_sync(0xffffffffu, second, o);
            if (ob < best) {
                second = min(best, os);
                best = ob;
            } else {
                second = min(second, ob);
            }
        }
        if (best == ~0ull) continue;
        const int bestDist = (int)(best >> 40);
        const int bestIdx = (int)(best & 0xFFFFF);
        const int bestLevel = g.kps[bestIdx].octave;
        const int bestDist2 = second == ~0ull ? 256 : (int)(second >> 40);
        const int bestLevel2 = second == ~0ull ? -1 : g.kps[(int)(second & 0xFFFFF)].octave;
        if (bestDist <= ORBGPU_TH_HIGH) {
            if (bestLevel == bestLevel2 && (float)bestDist > __fmul_rn(nnratio, (float)bestDist2)) continue;
            if (lane == 0) match_out[bestIdx] = imp;
            nmatches++;
        }
        __syncwarp();
    }
    if (lane == 0) *nmatches_out = nmatches;
}

// Parallel resolution of the same search by fixed-point rounds (the scheme
// of the batched search): round r evaluates every map point against the
// claims of round r-1's results; when a round changes nothing the results
// equal the sequential ones.  Pre-claimed keypoints (match_out == -2) are
// always excluded.  k_proj_resolve replays serially if no round converged.
__global__ void k_proj_round(GridDev g, int m, int slot_cap, const long long* start, const int* slot_count,
                             const uint64_t* slots, float nnratio, int round, int* claims3, int* res, int* changed, const int* pre) {
    const int lane = threadIdx.x & 31;
    const int local = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int nwarps = gridDim.x * (blockDim.x >> 5);
    if (round > 0 && changed[round - 1] == 0) return;
    const int n = g.n;
    int* claims_r = claims3 + (size_t)((round + 0) % 3) * n;
    int* claims_w = claims3 + (size_t)((round + 1) % 3) * n;
    int* claims_z = claims3 + (size_t)((round + 2) % 3) * n;
    for (int i = local * 32 + lane; i < n; i += nwarps * 32) claims_z[i] = PROJ_NONE;
    if (local >= m) return;
    const int cnt = min(slot_count[local], slot_cap);
    const uint64_t* row = cand_row(slots, slot_cap, start, local);
    uint64_t best = ~0ull, second = ~0ull;
    for (int b = 0; b < cnt; b += 32) {
        uint64_t key = ~0ull;
        if (b + lane < cnt) {
            key = row[b + lane];
            const int idx = (int)(key & 0xFFFFF);
            if (pre[idx] == -2 || claims_r[idx] < local || (int)(key >> 40) >= 256) key = ~0ull;
        }
        if (key < best) {
            second = best;
            best = key;
        } else if (key < second) {
            second = key;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t ob = __shfl_xor_sync(0xffffffffu, best, o);
        const uint64_t os = __shfl_xor_sync(0xffffffffu, second, o);
        if (ob < best) {
            second = best < os ? best : os;
            best = ob;
        } else {
            second = second < ob ? second : ob;
        }
    }
    int r = -1;
    if (best != ~0ull) {
        const int bestDist = (int)(best >> 40);
        const int bestIdx = (int)(best & 0xFFFFF);
        const int bestLevel = g.kps[bestIdx].octave;
        const int bestDist2 = second == ~0ull ? 256 : (int)(second >> 40);
        const int bestLevel2 = second == ~0ull ? -1 : g.kps[(int)(second & 0xFFFFF)].octave;
        if (bestDist <= ORBGPU_TH_HIGH &&
            !(bestLevel == bestLevel2 && (float)bestDist > __fmul_rn(nnratio, (float)bestDist2)))
            r = bestIdx;
    }
    if (lane == 0) {
        if (res[local] != r) changed[round] = 1;
        res[local] = r;
        if (r >= 0) atomicMin(&claims_w[r], local);
    }
}

// Converged rounds: write the matches; otherwise leave match_out for the
// serial replay.
__global__ void k_proj_finish(int m, const int* changed, const int* res, int* match_out, int* nmatches_out) {
    if (changed[PROJ_ROUNDS - 1] != 0) return;
    int nm = 0;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int r = res[i];
        if (r >= 0) {
            match_out[r] = i;
            nm++;
        }
    }
    atomicAdd(nmatches_out, nm);
}

__global__ void k_init_match_out(const uint8_t* claimed, int n, int* match_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) match_out[i] = (claimed && claimed[i]) ? -2 : -1;
}

// ----------------------------------------------------------------- SearchByProjection(Frame, LastFrame)
// src/ORBmatcher.cc:1710-1879.  Per LastFrame map point (one warp): the pose
// algebra with the reference's rounding (3 x 3 float product accumulated in
// double and stored as float, then a float addition; 1.0 / z in double), the
// window over the current grid with the motion-dependent level range, the
// stereo gate, and the candidates whose distance can be accepted
// (<= TH_HIGH: with no ratio test the first minimum is the answer, and a
// minimum above TH_HIGH is rejected either way).
struct FrameMotionDev {
    float T[12];
    float fx, fy, cx, cy, bf;
    float maxX, maxY;
    int level_mode;  // 1 forward, 2 backward, 0 neither
};

__device__ __forceinline__ float pose_row(const float* row, float X0, float X1, float X2) {
    double s = __dadd_rn(0.0, __dmul_rn((double)row[0], (double)X0));
    s = __dadd_rn(s, __dmul_rn((double)row[1], (double)X1));
    s = __dadd_rn(s, __dmul_rn((double)row[2], (double)X2));
    return __fadd_rn(__double2float_rn(s), row[3]);
}

__global__ void k_pf_candidates(GridDev g, FrameMotionDev mo, const orbgpu_keypoint* last_kps,
                                const orbgpu_frame_mappoint* mps, const uint8_t* mp_desc, int m, float th,
                                const int* cand_start, int* cand_count, uint64_t* cand_out, int fill) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i >= m) return;
    const orbgpu_frame_mappoint mp = mps[i];
    int total = 0;
    const int oct = last_kps[i].octave;
    bool live = (mp.flags & ORBGPU_MP_PRESENT) && !(mp.flags & ORBGPU_MP_OUTLIER) && oct >= 0 && oct < 16;
    float u = 0.f, v = 0.f, invzc = 0.f;
    if (live) {
        const float xc = pose_row(mo.T, mp.x, mp.y, mp.z);
        const float yc = pose_row(mo.T + 4, mp.x, mp.y, mp.z);
        const float zc = pose_row(mo.T + 8, mp.x, mp.y, mp.z);
        invzc = __double2float_rn(__ddiv_rn(1.0, (double)zc));
        u = __fadd_rn(__fmul_rn(__fmul_rn(mo.fx, xc), invzc), mo.cx);
        v = __fadd_rn(__fmul_rn(__fmul_rn(mo.fy, yc), invzc), mo.cy);
        // a non-finite projection finds no grid cell in the reference
        live = !(invzc < 0.f) && isfinite(u) && isfinite(v) && !(u < g.minX || u > mo.maxX) &&
               !(v < g.minY || v > mo.maxY);
    }
    if (live) {
        const float radius = __fmul_rn(th, g.scale[oct]);
        int minL, maxL;
        if (mo.level_mode == 1) {
            minL = oct;
            maxL = -1;
        } else if (mo.level_mode == 2) {
            minL = 0;
            maxL = oct;
        } else {
            minL = oct - 1;
            maxL = oct + 1;
        }
        int x0, x1, y0, y1;
        if (area_cells(g, u, v, radius, x0, x1, y0, y1)) {
            const uint8_t* dmp = mp_desc + (size_t)i * 32;
            const float ur = __fsub_rn(u, __fmul_rn(mo.bf, invzc));
            warp_window_recs(g, x0, x1, y0, y1, [&](const GridRec& rec, bool valid) {
                const int idx = (int)rec.idx, c = rec.cell();
                bool ok = valid && in_area(rec, u, v, radius, minL, maxL);
                if (ok && g.uright && g.uright[idx] > 0) {
                    const float er = fabsf(__fsub_rn(ur, g.uright[idx]));
                    if (er > radius) ok = false;
                }
                int dist = 256;
                if (ok) {
                    dist = hamming256_ptr(dmp, g.desc + (size_t)idx * 32);
                    ok = dist <= ORBGPU_TH_HIGH;
                }
                const unsigned msk = __ballot_sync(0xffffffffu, ok);
                if (fill && ok) {
                    const int pos = cand_start[i] + total + __popc(msk & ((1u << lane) - 1));
                    cand_out[pos] = cand_key(dist, c, idx);
                }
                total += __popc(msk);
            });
        }
    }
    if (!fill && lane == 0) cand_count[i] = total;
}

// ----------------------------------------------------------------- SearchByProjection(Frame, KeyFrame)
// src/ORBmatcher.cc:1891-2010 (relocalisation): the keyframe's map points
// that are usable (not NULL, not bad, not in sAlreadyFound) in keyframe order.
// Per map point (one warp): Rcw * X + tcw as in the frame-to-frame search
// (no depth test here), the projection, the distance invariance, the level
// MapPoint::PredictScale gives (thresholds of orbgpu_frustum_frame_init), the
// window of levels level - 1 .. level + 1 with radius th * scale[level], and
// the candidates at distance <= ORBdist (no ratio test: the first minimum is
// the answer, and a minimum above ORBdist is rejected either way).
struct KeyframeProjDev {
    float T[12];
    float Ow[3];
    float fx, fy, cx, cy;
    float maxX, maxY;
    int nlevels;
    float level_above[15];
    int orbdist;
    // 1: SearchByProjection(KeyFrame*, Scw, vpPoints, vpMatched, th)
    // (src/ORBmatcher.cc:423-560): depth test, IsInImage bounds, viewing angle,
    // levels level - 1 .. level, u = fx * (x * invz) + cx
    int sim3;
    // with sim3: Fuse(KeyFrame*, vpMapPoints, th) (src/ORBmatcher.cc:1107-1245)
    // adds the reprojection-error gate of every candidate (stereo with ur)
    int fuse;
    float bf;
    float inv_sigma2[16];
    // Fuse(KeyFrame*, Scw, ...) (src/ORBmatcher.cc:1290-1380): invz = 1.0 / z
    // in double, rounded to float
    int invz_double;
    // SearchBySim3 (src/ORBmatcher.cc:1441-1640): a second transform T2
    // applied to the camera coordinates (the Sim3 between the keyframes), the
    // depth for the distance invariance is |p3Dc| and there is no viewing
    // angle test
    int chain;
    float T2[12];
};

__global__ void k_pkf_candidates(GridDev g, KeyframeProjDev kp, const orbgpu_mappoint_geometry* mps,
                                 const uint8_t* usable, const uint8_t* mp_desc, int m, float th,
                                 const int* cand_start, int* cand_count, uint64_t* cand_out, int fill) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i >= m) return;
    int total = 0;
    bool live = usable[i] == 1;
    float u = 0.f, v = 0.f, ur_f = 0.f;
    int level = 0;
    if (live) {
        const orbgpu_mappoint_geometry mp = mps[i];
        float xc = pose_row(kp.T, mp.x, mp.y, mp.z);
        float yc = pose_row(kp.T + 4, mp.x, mp.y, mp.z);
        float zc = pose_row(kp.T + 8, mp.x, mp.y, mp.z);
        if (kp.chain) {
            const float x1 = xc, y1 = yc, z1 = zc;
            xc = pose_row(kp.T2, x1, y1, z1);
            yc = pose_row(kp.T2 + 4, x1, y1, z1);
            zc = pose_row(kp.T2 + 8, x1, y1, z1);
        }
        if (kp.sim3) {
            const float invz = kp.invz_double ? __double2float_rn(__ddiv_rn(1.0, (double)zc)) : __fdiv_rn(1.0f, zc);
            u = __fadd_rn(__fmul_rn(kp.fx, __fmul_rn(xc, invz)), kp.cx);
            v = __fadd_rn(__fmul_rn(kp.fy, __fmul_rn(yc, invz)), kp.cy);
            ur_f = __fsub_rn(u, __fmul_rn(kp.bf, invz));
            // KeyFrame::IsInImage (upper bounds exclusive); NaN fails it
            live = !(zc < 0.0f) && u >= g.minX && u < kp.maxX && v >= g.minY && v < kp.maxY;
        } else {
            const float invzc = __double2float_rn(__ddiv_rn(1.0, (double)zc));
            u = __fadd_rn(__fmul_rn(__fmul_rn(kp.fx, xc), invzc), kp.cx);
            v = __fadd_rn(__fmul_rn(__fmul_rn(kp.fy, yc), invzc), kp.cy);
            // a non-finite projection finds no grid cell in the reference
            live = isfinite(u) && isfinite(v) && !(u < g.minX || u > kp.maxX) && !(v < g.minY || v > kp.maxY);
        }
        if (live) {
            // PO = X - Ow, or the camera coordinates themselves for SearchBySim3
            const float po0 = kp.chain ? xc : __fsub_rn(mp.x, kp.Ow[0]);
            const float po1 = kp.chain ? yc : __fsub_rn(mp.y, kp.Ow[1]);
            const float po2 = kp.chain ? zc : __fsub_rn(mp.z, kp.Ow[2]);
            double ss = __dmul_rn((double)po0, (double)po0);
            ss = __dadd_rn(ss, __dmul_rn((double)po1, (double)po1));
            ss = __dadd_rn(ss, __dmul_rn((double)po2, (double)po2));
            const float dist = (float)__dsqrt_rn(ss);
            live = !(dist < __fmul_rn(0.8f, mp.min_distance) || dist > __fmul_rn(1.2f, mp.max_distance));
            if (live && kp.sim3 && !kp.chain) {
                // PO.dot(Pn) < 0.5 * dist, in double
                double dp = __dmul_rn((double)po0, (double)mp.nx);
                dp = __dadd_rn(dp, __dmul_rn((double)po1, (double)mp.ny));
                dp = __dadd_rn(dp, __dmul_rn((double)po2, (double)mp.nz));
                live = !(dp < __dmul_rn(0.5, (double)dist));
            }
            const float ratio = __fdiv_rn(mp.max_distance, dist);
            for (int n = 0; n < kp.nlevels - 1; n++) level += ratio > kp.level_above[n] ? 1 : 0;
        }
    }
    if (live) {
        const float radius = __fmul_rn(th, g.scale[level]);
        int x0, x1, y0, y1;
        if (area_cells(g, u, v, radius, x0, x1, y0, y1)) {
            const uint8_t* dmp = mp_desc + (size_t)i * 32;
            warp_window_recs(g, x0, x1, y0, y1, [&](const GridRec& rec, bool valid) {
                const int idx = (int)rec.idx, c = rec.cell();
                bool ok;
                if (kp.sim3) {
                    // KeyFrame::GetFeaturesInArea (src/KeyFrame.cc:785-830): a square
                    // window (|dx| < r and |dy| < r; Frame's is a disc), then the
                    // levels predicted - 1 .. predicted
                    ok = valid && rec.octave() >= level - 1 && rec.octave() <= level &&
                         fabsf(__fsub_rn(rec.x, u)) < radius && fabsf(__fsub_rn(rec.y, v)) < radius;
                } else {
                    ok = valid && in_area(rec, u, v, radius, level - 1, level + 1);
                }
                if (ok && kp.fuse) {
                    // chi-square gates of Fuse: 7.8 with the right coordinate, 5.99 without
                    const float ex = __fsub_rn(u, rec.x), ey = __fsub_rn(v, rec.y);
                    float e2 = __fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey));
                    const bool stereo = g.uright && g.uright[idx] >= 0.0f;
                    if (stereo) {
                        const float er = __fsub_rn(ur_f, g.uright[idx]);
                        e2 = __fadd_rn(e2, __fmul_rn(er, er));
                    }
                    ok = !((double)__fmul_rn(e2, kp.inv_sigma2[rec.octave() & 15]) > (stereo ? 7.8 : 5.99));
                }
                int dist = 256;
                if (ok) {
                    dist = hamming256_ptr(dmp, g.desc + (size_t)idx * 32);
                    ok = dist <= kp.orbdist;
                }
                const unsigned msk = __ballot_sync(0xffffffffu, ok);
                if (fill && ok) {
                    const int pos = cand_start[i] + total + __popc(msk & ((1u << lane) - 1));
                    cand_out[pos] = cand_key(dist, c, idx);
                }
                total += __popc(msk);
            });
        }
    }
    if (!fill && lane == 0) cand_count[i] = total;
}

// Fixed-point round r of the in-order assignment: map point i takes its
// first minimum among candidates not held by an observed map point j < i of
// round r-1's results (an owner without observations blocks nothing,
// src/ORBmatcher.cc:1800-1802; with mps NULL every owner blocks, as in
// SearchByProjection(Frame&, KeyFrame*, ...)).  A round that changes nothing
// equals the sequential result.
__global__ void k_pf_round(int n, int m, const int* cand_start, const int* cand_count, const uint64_t* cands,
                           const orbgpu_frame_mappoint* mps, int round, int* claims3, int* res, int* changed,
                           const int* pre) {
    const int lane = threadIdx.x & 31;
    const int local = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int nwarps = gridDim.x * (blockDim.x >> 5);
    if (round > 0 && changed[round - 1] == 0) return;
    int* claims_r = claims3 + (size_t)((round + 0) % 3) * n;
    int* claims_w = claims3 + (size_t)((round + 1) % 3) * n;
    int* claims_z = claims3 + (size_t)((round + 2) % 3) * n;
    for (int k = local * 32 + lane; k < n; k += nwarps * 32) claims_z[k] = PROJ_NONE;
    if (local >= m) return;
    const int s = cand_start[local], cnt = cand_count[local];
    uint64_t best = ~0ull;
    for (int b = lane; b < cnt; b += 32) {
        const uint64_t key = cands[s + b];
        const int idx = (int)(key & 0xFFFFF);
        if (pre[idx] != -2 && !(claims_r[idx] < local) && key < best) best = key;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t ob = __shfl_xor_sync(0xffffffffu, best, o);
        best = ob < best ? ob : best;
    }
    const int r = best == ~0ull ? -1 : (int)(best & 0xFFFFF);
    if (lane == 0) {
        if (res[local] != r) changed[round] = 1;
        res[local] = r;
        if (r >= 0 && (!mps || (mps[local].flags & ORBGPU_MP_OBSERVED))) atomicMin(&claims_w[r], local);
    }
}

// Sequential assignment when no round converged (one warp).
__global__ void k_pf_serial(int n, int m, const int* cand_start, const int* cand_count, const uint64_t* cands,
                            const orbgpu_frame_mappoint* mps, const int* changed, int* res, int* blocked,
                            const int* pre) {
    if (changed[PROJ_ROUNDS - 1] == 0) return;
    const int lane = threadIdx.x;
    for (int k = lane; k < n; k += 32) blocked[k] = pre[k] == -2;
    __syncwarp();
    for (int i = 0; i < m; i++) {
        const int s = cand_start[i], cnt = cand_count[i];
        uint64_t best = ~0ull;
        for (int b = lane; b < cnt; b += 32) {
            const uint64_t key = cands[s + b];
            if (!blocked[(int)(key & 0xFFFFF)] && key < best) best = key;
        }
        for (int o = 16; o > 0; o >>= 1) {
            const uint64_t ob = __shfl_xor_sync(0xffffffffu, best, o);
            best = ob < best ? ob : best;
        }
        const int r = best == ~0ull ? -1 : (int)(best & 0xFFFFF);
        if (lane == 0) {
            res[i] = r;
            if (r >= 0 && (!mps || (mps[i].flags & ORBGPU_MP_OBSERVED))) blocked[r] = 1;
        }
        __syncwarp();
    }
}

// Owners (the last map point that assigned each keypoint), the rotation
// histogram of every assignment (src/ORBmatcher.cc:1847-1857), the three
// maxima and the resets (:1862-1876), and the output codes.  One block.
__global__ void __launch_bounds__(1024) k_pf_finish(int n, int m, const int* res, const orbgpu_keypoint* last_kps,
                                                    const orbgpu_keypoint* cur_kps, int check_ori, int* owner,
                                                    int* bin_of, int* nulled, int* match_out, int* nmatches_out) {
    __shared__ int hist[ORBGPU_HISTO_LENGTH];
    __shared__ int s_nm, s_ind[3];
    if (threadIdx.x < ORBGPU_HISTO_LENGTH) hist[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_nm = 0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        owner[k] = -1;
        nulled[k] = 0;
    }
    __syncthreads();
    const float factor = __fdiv_rn((float)ORBGPU_HISTO_LENGTH, 360.0f);
    int nm = 0;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int r = res[i];
        int bin = -1;
        if (r >= 0) {
            nm++;
            atomicMax(&owner[r], i);
            if (check_ori) {
                float rot = __fsub_rn(last_kps[i].angle, cur_kps[r].angle);
                if (rot < 0.0f) rot = __fadd_rn(rot, 360.0f);
                bin = (int)roundf(__fmul_rn(rot, factor));
                if (bin == ORBGPU_HISTO_LENGTH) bin = 0;
                atomicAdd(&hist[bin], 1);
            }
        }
        bin_of[i] = bin;
    }
    atomicAdd(&s_nm, nm);
    __syncthreads();
    if (threadIdx.x == 0) {
        int ind1 = -1, ind2 = -1, ind3 = -1;
        if (check_ori) {
            int max1 = 0, max2 = 0, max3 = 0;
            for (int b = 0; b < ORBGPU_HISTO_LENGTH; b++) {  // ComputeThreeMaxima, src/ORBmatcher.cc:2035-2077
                const int sz = hist[b];
                if (sz > max1) {
                    max3 = max2; max2 = max1; max1 = sz;
                    ind3 = ind2; ind2 = ind1; ind1 = b;
                } else if (sz > max2) {
                    max3 = max2; max2 = sz;
                    ind3 = ind2; ind2 = b;
                } else if (sz > max3) {
                    max3 = sz;
                    ind3 = b;
                }
            }
            if ((float)max2 < __fmul_rn(0.1f, (float)max1)) {
                ind2 = -1;
                ind3 = -1;
            } else if ((float)max3 < __fmul_rn(0.1f, (float)max1)) {
                ind3 = -1;
            }
        }
        s_ind[0] = ind1;
        s_ind[1] = ind2;
        s_ind[2] = ind3;
    }
    __syncthreads();
    if (check_ori) {
        int removed = 0;
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const int b = bin_of[i];
            if (b < 0 || b == s_ind[0] || b == s_ind[1] || b == s_ind[2]) continue;
            nulled[res[i]] = 1;
            removed++;
        }
        atomicSub(&s_nm, removed);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int pre = match_out[k];
        match_out[k] = nulled[k] ? -4 : owner[k] >= 0 ? owner[k] : pre;
    }
    if (threadIdx.x == 0) *nmatches_out = s_nm;
}

// ----------------------------------------------------------------- stereo
// (the device functions are in orbgpu_stereo.cuh)
__global__ void __launch_bounds__(STEREO_INDEX_THREADS) k_stereo_index(const orbgpu_keypoint* kpsR, int nR, int nlevels,
                                                                       int nRows, int* start, uint4* recs,
                                                                       int* status) {
    if (threadIdx.x == 0) *status = 0;
    stereo_index_block(kpsR, nR, nlevels, nRows, start, recs);
}

__global__ void __launch_bounds__(32 * STEREO_WARPS) k_stereo_match(const orbgpu_keypoint* kpsL, const uint8_t* descL,
                                                                    int nL, const uint8_t* descR,
                                                                    const __grid_constant__ StereoLevels lv, int nRows,
                                                                    const int* start, const uint4* recs, float bf,
                                                                    float fx, float* uright, float* depth, int* sad,
                                                                    int* status) {
    const int iL = blockIdx.x * STEREO_WARPS + (threadIdx.x >> 5);
    if (iL < nL)
        stereo_match_warp(iL, kpsL, descL, descR, lv, nRows, start, recs, bf, fx, uright, depth, sad, status);
}

__global__ void __launch_bounds__(STEREO_INDEX_THREADS) k_stereo_median(int nL, const int* sad, float* uright, float* depth) {
    stereo_median_block(nL, sad, uright, depth);
}

// ----------------------------------------------------------------- distance batch
__global__ void k_descriptor_distance(const uint8_t* a, const uint8_t* b, int n, int* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = hamming256_ptr(a + (size_t)i * 32, b + (size_t)i * 32);
}

}  // namespace orbgpu

using namespace orbgpu;

// ----------------------------------------------------------------- host side
struct orbgpu_matcher {
    float nnratio;
    int check_ori;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    // scratch (grown on demand)
    void* scratch = nullptr;
    size_t scratch_bytes = 0;
    int* h_pinned = nullptr;
    // kNN workspaces that no call holds (KnnWorkspace)
    std::mutex knn_mutex;
    orbgpu::KnnBuffers* knn_work = nullptr;
    size_t knn_kept = 0;  // their bytes
};

namespace {

struct Staged {
    const orbgpu_keypoint* kps = nullptr;
    const uint8_t* desc = nullptr;
    const float* uright = nullptr;
};

struct Bump {
    uint8_t* base;
    size_t off = 0, cap;
    template <typename T> T* take(size_t n) {
        off = (off + 255) & ~(size_t)255;
        T* p = (T*)(base + off);
        off += n * sizeof(T);
        return p;
    }
};

int ensure_scratch(orbgpu_matcher* m, size_t bytes) {
    if (bytes <= m->scratch_bytes) return ORBGPU_OK;
    ORBGPU_CUDA_TRY(cudaStreamSynchronize(m->stream));
    if (m->scratch) cudaFree(m->scratch);
    m->scratch = nullptr;
    m->scratch_bytes = 0;
    ORBGPU_CUDA_TRY(cudaMalloc(&m->scratch, bytes));
    m->scratch_bytes = bytes;
    return ORBGPU_OK;
}

// Device copies of a frame's arrays (or the caller's device pointers).
int stage_frame(orbgpu_matcher* m, const orbgpu_frame* f, Bump& b, Staged& s) {
    if (f->mem == ORBGPU_MEM_DEVICE) {
        s.kps = f->keypoints;
        s.desc = f->descriptors;
        s.uright = f->uright;
        return ORBGPU_OK;
    }
    orbgpu_keypoint* k = b.take<orbgpu_keypoint>(std::max(1, f->n));
    uint8_t* d = b.take<uint8_t>((size_t)std::max(1, f->n) * 32);
    if (f->n > 0) {
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(k, f->keypoints, sizeof(orbgpu_keypoint) * f->n, cudaMemcpyHostToDevice, m->stream));
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(d, f->descriptors, 32 * (size_t)f->n, cudaMemcpyHostToDevice, m->stream));
    }
    s.kps = k;
    s.desc = d;
    s.uright = nullptr;
    if (f->uright) {
        float* u = b.take<float>(std::max(1, f->n));
        if (f->n > 0) ORBGPU_CUDA_TRY(cudaMemcpyAsync(u, f->uright, sizeof(float) * f->n, cudaMemcpyHostToDevice, m->stream));
        s.uright = u;
    }
    return ORBGPU_OK;
}

size_t frame_stage_bytes(const orbgpu_frame* f) {
    if (f->mem == ORBGPU_MEM_DEVICE) return 0;
    return (size_t)std::max(1, f->n) * (sizeof(orbgpu_keypoint) + 32 + 4) + 1024;
}

size_t grid_bytes(int n) { return (size_t)(3 * ORBGPU_GRID_CELLS + 8) * sizeof(int) + (size_t)std::max(1, n) * sizeof(GridRec) + 2048; }

// AssignFeaturesToGrid (src/Frame.cc:399-423) on the device.
int build_grid(orbgpu_matcher* m, const orbgpu_frame* f, const Staged& s, Bump& b, GridDev& g) {
    int* cell_start = b.take<int>(ORBGPU_GRID_CELLS + 1);
    GridRec* recs = b.take<GridRec>(std::max(1, f->n));
    g.kps = s.kps;
    g.desc = s.desc;
    g.uright = s.uright;
    g.n = f->n;
    g.minX = 0.0f;
    g.minY = 0.0f;
    g.invW = static_cast<float>(ORBGPU_GRID_COLS) / static_cast<float>((float)f->width - 0.0f);
    g.invH = static_cast<float>(ORBGPU_GRID_ROWS) / static_cast<float>((float)f->height - 0.0f);
    g.cell_start = cell_start;
    g.recs = recs;
    for (int l = 0; l < 16; l++) g.scale[l] = l < f->nlevels ? f->scale_factors[l] : 1.0f;
    if (f->n <= GRID_BLOCK_N) {
        k_grid_build<<<1, 1024, 0, m->stream>>>(s.kps, f->n, g.minX, g.minY, g.invW, g.invH, cell_start, recs);
    } else {
        int* cell_count = b.take<int>(ORBGPU_GRID_CELLS);
        int* cursor = b.take<int>(ORBGPU_GRID_CELLS);
        const int blocks = (f->n + 255) / 256;
        ORBGPU_CUDA_TRY(cudaMemsetAsync(cell_count, 0, sizeof(int) * ORBGPU_GRID_CELLS, m->stream));
        k_grid_count<<<blocks, 256, 0, m->stream>>>(s.kps, f->n, g.minX, g.minY, g.invW, g.invH, cell_count);
        k_grid_scan<<<1, 1024, 0, m->stream>>>(cell_count, cell_start, cursor);
        k_grid_fill<<<blocks, 256, 0, m->stream>>>(s.kps, f->n, g.minX, g.minY, g.invW, g.invH, cursor, recs);
    }
    ORBGPU_CUDA_TRY(cudaGetLastError());
    return ORBGPU_OK;
}

bool frame_ok(const orbgpu_frame* f) {
    return f && f->n >= 0 && f->n < (1 << 20) && f->width > 0 && f->height > 0 && f->nlevels >= 1 &&
           f->nlevels <= 16 && (f->n == 0 || (f->keypoints && f->descriptors));
}

}  // namespace

KnnWorkspace::~KnnWorkspace() {
    if (!b) return;
    std::lock_guard<std::mutex> lock(m->knn_mutex);
    if (m->knn_kept + b->bytes > KNN_KEEP_BYTES) b->drop(m->stream);
    m->knn_kept += b->bytes;
    b->next = m->knn_work;
    m->knn_work = b;
}
int KnnWorkspace::take(size_t need) {
    {
        std::lock_guard<std::mutex> lock(m->knn_mutex);
        // the smallest that is large enough, else the largest
        KnnBuffers** best = &m->knn_work;
        for (KnnBuffers** p = best; *p; p = &(*p)->next)
            if ((*best)->bytes < need ? (*p)->bytes > (*best)->bytes : (*p)->bytes >= need && (*p)->bytes < (*best)->bytes)
                best = p;
        b = *best;
        if (b) {
            *best = b->next;
            m->knn_kept -= b->bytes;
        }
    }
    if (!b) {
        KnnBuffers* fresh = new (std::nothrow) KnnBuffers();
        if (!fresh || cudaMallocHost(&fresh->pinned, 64) != cudaSuccess) {
            delete fresh;
            orbgpu_set_last_error("page-locked allocation failed", __FILE__, __LINE__);
            return ORBGPU_ERR_OOM;
        }
        b = fresh;
    }
    if (b->bytes >= need) return ORBGPU_OK;
    b->drop(m->stream);
    ORBGPU_CUDA_TRY(cudaMallocAsync((void**)&b->data, need, m->stream));
    b->bytes = need;
    return ORBGPU_OK;
}

extern "C" int orbgpu_matcher_create(float nnratio, int check_orientation, void* stream, orbgpu_matcher** out) {
    if (!out) return ORBGPU_ERR_BAD_ARG;
    int dev;
    ORBGPU_CUDA_TRY(cudaGetDevice(&dev));
    orbgpu_matcher* m = new orbgpu_matcher();
    m->nnratio = nnratio;
    m->check_ori = check_orientation;
    if (stream) m->stream = (cudaStream_t)stream;
    else {
        if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) {
            delete m;
            return ORBGPU_ERR_CUDA;
        }
        m->own_stream = true;
    }
    if (cudaMallocHost(&m->h_pinned, 64) != cudaSuccess) {
        orbgpu_matcher_destroy(m);
        return ORBGPU_ERR_OOM;
    }
    *out = m;
    return ORBGPU_OK;
}

extern "C" int orbgpu_matcher_destroy(orbgpu_matcher* m) {
    if (!m) return ORBGPU_OK;
    if (m->stream) cudaStreamSynchronize(m->stream);
    cudaFree(m->scratch);
    cudaFreeHost(m->h_pinned);
    while (KnnBuffers* w = m->knn_work) {
        m->knn_work = w->next;
        w->drop(m->stream);
        cudaFreeHost(w->pinned);
        delete w;
    }
    if (m->own_stream) cudaStreamDestroy(m->stream);
    delete m;
    return ORBGPU_OK;
}

// Runs the two-pass candidate listing: count, scan, fill.  Returns the
// device candidate arrays in (start, count, keys).
template <typename Launch>
static int candidate_lists(orbgpu_matcher* m, int nq, Bump& b, Launch launch, int*& start, int*& count,
                           uint64_t*& keys, int& total) {
    count = b.take<int>(std::max(1, nq));
    start = b.take<int>(std::max(1, nq));
    int* d_total = b.take<int>(1);
    launch((const int*)nullptr, count, (uint64_t*)nullptr, 0);
    k_exclusive_scan<<<1, 1024, 0, m->stream>>>(count, nq, start, d_total);
    ORBGPU_CUDA_TRY(cudaMemcpyAsync(m->h_pinned, d_total, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    ORBGPU_CUDA_TRY(cudaStreamSynchronize(m->stream));
    total = m->h_pinned[0];
    const size_t need = b.off + 256 + sizeof(uint64_t) * (size_t)std::max(1, total);
    if (need > b.cap) return ORBGPU_ERR_CAPACITY;
    keys = b.take<uint64_t>(std::max(1, total));
    launch((const int*)start, count, keys, 1);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    return ORBGPU_OK;
}

// The candidate rows of a search's nq queries (cand_row): of 64 keys, widened
// where a window holds more; rows of the queries' own lengths where a few
// crowded windows would make wide rows take more than CAND_ROWS_BYTES.
#define CAND_ROWS_BYTES ((size_t)1 << 30)
struct CandRows {
    int cap = 64;
    std::vector<long long> start;  // empty: rows of 'cap' keys
    size_t keys;                   // in all rows

    explicit CandRows(int nq) : keys((size_t)64 * nq) {}
    // after a call whose longest row was 'longest'; count: the queries' candidates (device)
    int widen(orbgpu_matcher* m, int nq, int longest, const int* count, size_t key_bytes, bool own_lengths) {
        cap = (longest + 63) / 64 * 64;
        keys = (size_t)nq * cap;
        if (!own_lengths || keys * key_bytes <= CAND_ROWS_BYTES) return ORBGPU_OK;
        std::vector<int> n(nq);
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(n.data(), count, sizeof(int) * nq, cudaMemcpyDeviceToHost, m->stream));
        ORBGPU_CUDA_TRY(cudaStreamSynchronize(m->stream));
        start.resize(nq);
        keys = 0;
        for (int i = 0; i < nq; i++) {
            start[i] = (long long)keys;
            keys += n[i];
        }
        return ORBGPU_OK;
    }
    size_t bytes(size_t key_bytes) const { return key_bytes * std::max<size_t>(1, keys) + sizeof(long long) * start.size() + 512; }
    int stage(orbgpu_matcher* m, Bump& b, const long long** d_start) const {
        *d_start = nullptr;
        if (start.empty()) return ORBGPU_OK;
        long long* d = b.take<long long>(start.size());
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(d, start.data(), sizeof(long long) * start.size(), cudaMemcpyHostToDevice, m->stream));
        *d_start = d;
        return ORBGPU_OK;
    }
};

extern "C" int orbgpu_search_for_initialization(orbgpu_matcher* m, const orbgpu_frame* f1, const orbgpu_frame* f2,
                                                float* prev_matched, int* matches12, int window_size, int* nmatches) {
    if (!m || !frame_ok(f1) || !frame_ok(f2) || !prev_matched || !matches12 || !nmatches) return ORBGPU_ERR_BAD_ARG;
    const int n1 = f1->n, n2 = f2->n;
    *nmatches = 0;
    for (int i = 0; i < n1; i++) matches12[i] = -1;
    if (n1 == 0) return ORBGPU_OK;
    CandRows rows(n1);
    for (int attempt = 0; attempt < 2; attempt++) {
        const size_t est = frame_stage_bytes(f1) + frame_stage_bytes(f2) + grid_bytes(n2) + (size_t)n1 * 5 * sizeof(int) +
                           init_resolve_bytes(n1, n2) + rows.bytes(sizeof(uint64_t)) + 16 * 1024;
        int rc = ensure_scratch(m, est);
        if (rc) return rc;
        Bump b{(uint8_t*)m->scratch, 0, m->scratch_bytes};
        Staged s1, s2;
        if ((rc = stage_frame(m, f1, b, s1)) || (rc = stage_frame(m, f2, b, s2))) return rc;
        GridDev g2;
        if ((rc = build_grid(m, f2, s2, b, g2))) return rc;
        float* d_prev = b.take<float>(2 * n1);
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(d_prev, prev_matched, sizeof(float) * 2 * n1, cudaMemcpyHostToDevice, m->stream));
        int* count = b.take<int>(n1);
        int* m12 = b.take<int>(n1);
        int* d_status = b.take<int>(2);  // most candidates of a keypoint, matches
        int* work = b.take<int>(init_resolve_bytes(n1, n2) / sizeof(int));
        uint64_t* slots = b.take<uint64_t>(std::max<size_t>(1, rows.keys));
        const long long* d_start;
        if ((rc = rows.stage(m, b, &d_start))) return rc;
        ORBGPU_CUDA_TRY(cudaMemsetAsync(d_status, 0, 2 * sizeof(int), m->stream));
        const int wpb = 8;
        k_init_candidates<<<(n1 + wpb - 1) / wpb, 32 * wpb, 0, m->stream>>>(g2, s1.kps, s1.desc, n1, d_prev,
                                                                         (float)window_size, m->nnratio, rows.cap, d_start,
                                                                         slots, count, d_status);
        // the resolution's arrays in shared memory up to 200 KiB (8,500
        // keypoints a frame), else in the scratch
        const int local = init_resolve_bytes(n1, n2) <= 200 * 1024;
        ORBGPU_CUDA_TRY(allow_max_dynamic_smem(k_init_resolve));
        k_init_resolve<<<1, 1024, local ? init_resolve_bytes(n1, n2) : 0, m->stream>>>(
            s1.kps, n1, s2.kps, n2, rows.cap, d_start, count, slots, m->nnratio, m->check_ori, local, work, m12, d_status + 1);
        ORBGPU_CUDA_TRY(cudaGetLastError());
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(m->h_pinned, d_status, 2 * sizeof(int), cudaMemcpyDeviceToHost, m->stream));
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(matches12, m12, sizeof(int) * n1, cudaMemcpyDeviceToHost, m->stream));
        ORBGPU_CUDA_TRY(cudaStreamSynchronize(m->stream));
        if (m->h_pinned[0] > rows.cap) {  // a window held more candidates than a row: widen and redo
            if ((rc = rows.widen(m, n1, m->h_pinned[0], count, sizeof(uint64_t), true))) return rc;
            continue;
        }
        *nmatches = m->h_pinned[1];
        // vbPrevMatched update (src/ORBmatcher.cc:712-714)
        std::vector<orbgpu_keypoint> k2;
        if (f2->mem == ORBGPU_MEM_DEVICE) {
            k2.resize(n2);
            if (n2) ORBGPU_CUDA_TRY(cudaMemcpy(k2.data(), f2->keypoints, sizeof(orbgpu_keypoint) * n2, cudaMemcpyDeviceToHost));
        }
        const orbgpu_keypoint* K2 = f2->mem == ORBGPU_MEM_DEVICE ? k2.data() : f2->keypoints;
        for (int i1 = 0; i1 < n1; i1++)
            if (matches12[i1] >= 0) {
                prev_matched[2 * i1] = K2[matches12[i1]].x;
                prev_matched[2 * i1 + 1] = K2[matches12[i1]].y;
            }
        return ORBGPU_OK;
    }
    return ORBGPU_ERR_CAPACITY;
}

extern "C" int orbgpu_search_by_projection(orbgpu_matcher* m, const orbgpu_frame* f, const orbgpu_mappoint* mappoints,
                                           const uint8_t* mp_descriptors, int n_mappoints, float th,
                                           const uint8_t* claimed, int* match_out, int mem, int* nmatches) {
    if (!m || !frame_ok(f) || n_mappoints < 0 || (n_mappoints > 0 && (!mappoints || !mp_descriptors)) || !match_out ||
        !nmatches)
        return ORBGPU_ERR_BAD_ARG;
    const int n = f->n, M = n_mappoints;
    *nmatches = 0;
    // in one block with 32-bit keys when the frame fits in shared memory, else
    // with 64-bit keys in global-memory rounds
    const bool smem = n < ORBGPU_KEY32_MAX_N && proj_resolve_smem(n, M) <= 200 * 1024;
    const size_t key_bytes = smem ? sizeof(uint32_t) : sizeof(uint64_t);
    CandRows rows(M);
    for (int attempt = 0; attempt < 2; attempt++) {
        const size_t est = frame_stage_bytes(f) + grid_bytes(n) + (size_t)std::max(1, M) * (sizeof(orbgpu_mappoint) + 32 + 16) +
                           rows.bytes(key_bytes) + (size_t)std::max(1, n) * 24 + 64 * 1024;
        int rc = ensure_scratch(m, est);
        if (rc) return rc;
        Bump b{(uint8_t*)m->scratch, 0, m->scratch_bytes};
        Staged s;
        if ((rc = stage_frame(m, f, b, s))) return rc;
        GridDev g;
        if ((rc = build_grid(m, f, s, b, g))) return rc;
        const orbgpu_mappoint* d_mps = mappoints;
        const uint8_t* d_mpd = mp_descriptors;
        const uint8_t* d_claimed = claimed;
        int* d_match = match_out;
        if (mem != ORBGPU_MEM_DEVICE) {
            orbgpu_mappoint* a = b.take<orbgpu_mappoint>(std::max(1, M));
            uint8_t* dd = b.take<uint8_t>((size_t)std::max(1, M) * 32);
            if (M) {
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(a, mappoints, sizeof(orbgpu_mappoint) * M, cudaMemcpyHostToDevice, m->stream));
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(dd, mp_descriptors, 32 * (size_t)M, cudaMemcpyHostToDevice, m->stream));
            }
            d_mps = a;
            d_mpd = dd;
            if (claimed) {
                uint8_t* c = b.take<uint8_t>(std::max(1, n));
                if (n) ORBGPU_CUDA_TRY(cudaMemcpyAsync(c, claimed, n, cudaMemcpyHostToDevice, m->stream));
                d_claimed = c;
            }
            d_match = b.take<int>(std::max(1, n));
        }
        int* d_status = b.take<int>(3);  // most candidates of a map point, not converged, matches
        int* count = b.take<int>(std::max(1, M));
        void* slots = b.take<uint8_t>(key_bytes * std::max<size_t>(1, rows.keys));
        const long long* d_start;
        if ((rc = rows.stage(m, b, &d_start))) return rc;
        ORBGPU_CUDA_TRY(cudaMemsetAsync(d_status, 0, 3 * sizeof(int), m->stream));
        const int wpb = 8, mpb = wpb * (32 / PROJ_SEG);
        if (smem) {
            if (M > 0)
                k_proj_candidates<uint32_t><<<(M + mpb - 1) / mpb, 32 * wpb, 0, m->stream>>>(
                    g, d_mps, d_mpd, M, th, m->nnratio, rows.cap, d_start, (uint32_t*)slots, count, d_status);
            ORBGPU_CUDA_TRY(allow_max_dynamic_smem(k_proj_resolve_smem));
            k_proj_resolve_smem<<<1, 1024, proj_resolve_smem(n, M), m->stream>>>(
                s.kps, n, M, (const uint32_t*)slots, rows.cap, count, m->nnratio, d_claimed, d_match, d_status + 2, d_status);
        } else {
            if (M > 0)
                k_proj_candidates<uint64_t><<<(M + mpb - 1) / mpb, 32 * wpb, 0, m->stream>>>(
                    g, d_mps, d_mpd, M, th, m->nnratio, rows.cap, d_start, (uint64_t*)slots, count, d_status);
            if (n > 0) k_init_match_out<<<(n + 255) / 256, 256, 0, m->stream>>>(d_claimed, n, d_match);
            int* claims3 = b.take<int>((size_t)3 * std::max(1, n));
            int* res = b.take<int>(std::max(1, M));
            int* changed = b.take<int>(PROJ_ROUNDS);
            ORBGPU_CUDA_TRY(cudaMemsetAsync(claims3, 0x7f, sizeof(int) * (size_t)3 * std::max(1, n), m->stream));
            ORBGPU_CUDA_TRY(cudaMemsetAsync(res, 0xfe, sizeof(int) * std::max(1, M), m->stream));
            ORBGPU_CUDA_TRY(cudaMemsetAsync(changed, 0, sizeof(int) * PROJ_ROUNDS, m->stream));
            if (M > 0) {
                const int warps = std::max(M, (n + 31) / 32);
                for (int r = 0; r < PROJ_ROUNDS; r++)
                    k_proj_round<<<(warps + wpb - 1) / wpb, 32 * wpb, 0, m->stream>>>(
                        g, M, rows.cap, d_start, count, (const uint64_t*)slots, m->nnratio, r, claims3, res, changed, d_match);
                k_proj_finish<<<1, 256, 0, m->stream>>>(M, changed, res, d_match, d_status + 2);
                k_proj_resolve<<<1, 32, 0, m->stream>>>(g, M, rows.cap, d_start, count, (const uint64_t*)slots, m->nnratio,
                                                        d_match, d_status + 2, changed);
            }
        }
        ORBGPU_CUDA_TRY(cudaGetLastError());
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(m->h_pinned, d_status, 3 * sizeof(int), cudaMemcpyDeviceToHost, m->stream));
        if (mem != ORBGPU_MEM_DEVICE && n > 0)
            ORBGPU_CUDA_TRY(cudaMemcpyAsync(match_out, d_match, sizeof(int) * n, cudaMemcpyDeviceToHost, m->stream));
        ORBGPU_CUDA_TRY(cudaStreamSynchronize(m->stream));
        if (m->h_pinned[0] > rows.cap) {  // a window held more candidates than a row: widen and redo
            // (the one-block resolution reads rows of one length, of 4,095 keys at most)
            if ((rc = rows.widen(m, M, m->h_pinned[0], count, key_bytes, !smem))) return rc;
            continue;
        }
        if (m->h_pinned[1]) {
            orbgpu_set_last_error("projection search: resolution failed", __FILE__, __LINE__);
            return ORBGPU_ERR_CUDA;
        }
        *nmatches = m->h_pinned[2];
        return ORBGPU_OK;
    }
    return ORBGPU_ERR_CAPACITY;
}

// The reference's bForward / bBackward decision (src/ORBmatcher.cc:1724-1741):
// twc = -Rcw' tcw and tlc = Rlw twc + tlw with cv::Mat rounding (products
// accumulated in double, stored as float, then a float addition).
int orbgpu::motion_level_mode(const orbgpu_frame_motion& mo, int mono) {
    const float* T = mo.Tcw;
    const float tcw[3] = {T[3], T[7], T[11]};
    float twc[3];
    for (int r = 0; r < 3; r++) {
        const float col[3] = {-T[r], -T[4 + r], -T[8 + r]};
        double s = 0.0;
        for (int k = 0; k < 3; k++) s += (double)col[k] * (double)tcw[k];
        twc[r] = (float)s;
    }
    const float* L = mo.Tlw;
    double s = 0.0;
    for (int k = 0; k < 3; k++) s += (double)L[8 + k] * (double)twc[k];
    const float tlcz = (float)s + L[11];
    const bool fwd = tlcz > mo.b && !mono;
    const bool bwd = -tlcz > mo.b && !mono;
    return fwd ? 1 : bwd ? 2 : 0;
}

extern "C" int orbgpu_search_by_projection_frame(orbgpu_matcher* m, const orbgpu_frame* current,
                                                 const orbgpu_frame* last, const orbgpu_frame_mappoint* last_mappoints,
                                                 const uint8_t* last_mp_descriptors, const orbgpu_frame_motion* motion,
                                                 float th, int mono, const uint8_t* claimed, int* match_out, int mem,
                                                 int* nmatches) {
    if (!m || !frame_ok(current) || !last || last->n < 0 || last->n >= (1 << 20) || (last->n > 0 && !last->keypoints) ||
        !motion || !match_out || !nmatches || (last->n > 0 && (!last_mappoints || !last_mp_descriptors)))
        return ORBGPU_ERR_BAD_ARG;
    const int n = current->n, M = last->n;
    *nmatches = 0;
    const int mode = motion_level_mode(*motion, mono);
    FrameMotionDev mo;
    std::memcpy(mo.T, motion->Tcw, sizeof(mo.T));
    mo.fx = motion->fx;
    mo.fy = motion->fy;
    mo.cx = motion->cx;
    mo.cy = motion->cy;
    mo.bf = motion->bf;
    mo.maxX = (float)current->width;
    mo.maxY = (float)current->height;
    mo.level_mode = mode;
    size_t est = frame_stage_bytes(current) + grid_bytes(n) +
                 (size_t)std::max(1, M) * (sizeof(orbgpu_frame_mappoint) + sizeof(orbgpu_keypoint) + 32 + 32) +
                 (size_t)std::max(1, n) * 32 + 64 * 1024 + sizeof(uint64_t) * (size_t)std::max(1, M) * 32;
    for (int attempt = 0; attempt < 2; attempt++) {
        int rc = ensure_scratch(m, est);
        if (rc) return rc;
        Bump b{(uint8_t*)m->scratch, 0, m->scratch_bytes};
        Staged s;
        if ((rc = stage_frame(m, current, b, s))) return rc;
        GridDev g;
        if ((rc = build_grid(m, current, s, b, g))) return rc;
        const orbgpu_keypoint* d_lk = last->keypoints;
        if (last->mem != ORBGPU_MEM_DEVICE) {
            orbgpu_keypoint* k = b.take<orbgpu_keypoint>(std::max(1, M));
            if (M)
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(k, last->keypoints, sizeof(orbgpu_keypoint) * M, cudaMemcpyHostToDevice,
                                                m->stream));
            d_lk = k;
        }
        const orbgpu_frame_mappoint* d_mps = last_mappoints;
        const uint8_t* d_mpd = last_mp_descriptors;
        const uint8_t* d_claimed = claimed;
        int* d_match = match_out;
        if (mem != ORBGPU_MEM_DEVICE) {
            orbgpu_frame_mappoint* a = b.take<orbgpu_frame_mappoint>(std::max(1, M));
            uint8_t* dd = b.take<uint8_t>((size_t)std::max(1, M) * 32);
            if (M) {
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(a, last_mappoints, sizeof(orbgpu_frame_mappoint) * M,
                                                cudaMemcpyHostToDevice, m->stream));
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(dd, last_mp_descriptors, 32 * (size_t)M, cudaMemcpyHostToDevice,
                                                m->stream));
            }
            d_mps = a;
            d_mpd = dd;
            if (claimed) {
                uint8_t* c = b.take<uint8_t>(std::max(1, n));
                if (n) ORBGPU_CUDA_TRY(cudaMemcpyAsync(c, claimed, n, cudaMemcpyHostToDevice, m->stream));
                d_claimed = c;
            }
            d_match = b.take<int>(std::max(1, n));
        }
        if (n > 0) k_init_match_out<<<(n + 255) / 256, 256, 0, m->stream>>>(d_claimed, n, d_match);
        int *start, *count, total = 0;
        uint64_t* keys = nullptr;
        auto launch = [&](const int* st, int* cnt, uint64_t* out, int fill) {
            const int wpb = 8;
            if (M > 0)
                k_pf_candidates<<<(M + wpb - 1) / wpb, 32 * wpb, 0, m->stream>>>(g, mo, d_lk, d_mps, d_mpd, M, th, st,
                                                                              cnt, out, fill);
        };
        rc = candidate_lists(m, M, b, launch, start, count, keys, total);
        if (rc == ORBGPU_ERR_CAPACITY) {
            est = est + sizeof(uint64_t) * (size_t)total * 2;
            continue;
        }
        if (rc) return rc;
        int* d_nm = b.take<int>(1);
        int* claims3 = b.take<int>((size_t)3 * std::max(1, n));
        int* res = b.take<int>(std::max(1, M));
        int* changed = b.take<int>(PROJ_ROUNDS);
        int* owner = b.take<int>(std::max(1, n));
        int* nulled = b.take<int>(std::max(1, n));
        int* bin_of = b.take<int>(std::max(1, M));
        ORBGPU_CUDA_TRY(cudaMemsetAsync(d_nm, 0, sizeof(int), m->stream));
        ORBGPU_CUDA_TRY(cudaMemsetAsync(claims3, 0x7f, sizeof(int) * (size_t)3 * std::max(1, n), m->stream));
        ORBGPU_CUDA_TRY(cudaMemsetAsync(res, 0xfe, sizeof(int) * std::max(1, M), m->stream));
        ORBGPU_CUDA_TRY(cudaMemsetAsync(changed, 0, sizeof(int) * PROJ_ROUNDS, m->stream));
        if (M > 0 && n > 0) {
            const int wpb = 8;
            const int warps = std::max(M, (n + 31) / 32);
            for (int r = 0; r < PROJ_ROUNDS; r++)
                k_pf_round<<<(warps + wpb - 1) / wpb, 32 * wpb, 0, m->stream>>>(n, M, start, count, keys, d_mps, r,
                                                                              claims3, res, changed, d_match);
            k_pf_serial<<<1, 32, 0, m->stream>>>(n, M, start, count, keys, d_mps, changed, res, claims3, d_match);
            k_pf_finish<<<1, 1024, 0, m->stream>>>(n, M, res, d_lk, s.kps, m->check_ori, owner, bin_of, nulled, d_match,
                                                   d_nm);
        }
        ORBGPU_CUDA_TRY(cudaGetLastError());
        if (mem != ORBGPU_MEM_DEVICE && n > 0)
            ORBGPU_CUDA_TRY(cudaMemcpyAsync(match_out, d_match, sizeof(int) * n, cudaMemcpyDeviceToHost, m->stream));
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(m->h_pinned, d_nm, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
        ORBGPU_CUDA_TRY(cudaStreamSynchronize(m->stream));
        *nmatches = m->h_pinned[0];
        return ORBGPU_OK;
    }
    return ORBGPU_ERR_CAPACITY;
}

static int search_projection_keyframe(orbgpu_matcher* m, const orbgpu_frame* current, const KeyframeProjDev& kp,
                                      const orbgpu_keypoint* kf_keypoints, const orbgpu_mappoint_geometry* mappoints,
                                      const uint8_t* mp_descriptors, const uint8_t* usable, int n_kf, float th,
                                      const uint8_t* claimed, int* match_out, int mem, int* nmatches);

extern "C" int orbgpu_search_by_projection_keyframe(orbgpu_matcher* m, const orbgpu_frame* current,
                                                    const orbgpu_frustum_frame* pose,
                                                    const orbgpu_keypoint* kf_keypoints,
                                                    const orbgpu_mappoint_geometry* mappoints,
                                                    const uint8_t* mp_descriptors, const uint8_t* usable, int n_kf,
                                                    float th, int orbdist, const uint8_t* claimed, int* match_out,
                                                    int mem, int* nmatches) {
    if (!m || !frame_ok(current) || !pose || n_kf < 0 || n_kf >= (1 << 20) || !match_out || !nmatches ||
        (n_kf > 0 && (!kf_keypoints || !mappoints || !mp_descriptors || !usable)) || pose->nlevels < 1 ||
        pose->nlevels > 16)
        return ORBGPU_ERR_BAD_ARG;
    KeyframeProjDev kp;
    std::memset(&kp, 0, sizeof(kp));
    for (int r = 0; r < 3; r++) {
        for (int c = 0; c < 3; c++) kp.T[4 * r + c] = pose->Rcw[3 * r + c];
        kp.T[4 * r + 3] = pose->tcw[r];
        kp.Ow[r] = pose->Ow[r];
    }
    kp.fx = pose->fx;
    kp.fy = pose->fy;
    kp.cx = pose->cx;
    kp.cy = pose->cy;
    kp.maxX = (float)current->width;
    kp.maxY = (float)current->height;
    kp.nlevels = pose->nlevels;
    std::memcpy(kp.level_above, pose->level_above, sizeof(kp.level_above));
    kp.orbdist = orbdist;
    kp.sim3 = 0;
    return search_projection_keyframe(m, current, kp, kf_keypoints, mappoints, mp_descriptors, usable, n_kf, th,
                                      claimed, match_out, mem, nmatches);
}

// The candidate lists and in-order resolution shared by the relocalisation
// and the loop-closing projection searches.
static int search_projection_keyframe(orbgpu_matcher* m, const orbgpu_frame* current, const KeyframeProjDev& kp,
                                      const orbgpu_keypoint* kf_keypoints, const orbgpu_mappoint_geometry* mappoints,
                                      const uint8_t* mp_descriptors, const uint8_t* usable, int n_kf, float th,
                                      const uint8_t* claimed, int* match_out, int mem, int* nmatches) {
    const int n = current->n, M = n_kf;
    *nmatches = 0;
    size_t est = frame_stage_bytes(current) + grid_bytes(n) +
                 (size_t)std::max(1, M) * (sizeof(orbgpu_mappoint_geometry) + sizeof(orbgpu_keypoint) + 32 + 1 + 32) +
                 (size_t)std::max(1, n) * 32 + 64 * 1024 + sizeof(uint64_t) * (size_t)std::max(1, M) * 32;
    for (int attempt = 0; attempt < 2; attempt++) {
        int rc = ensure_scratch(m, est);
        if (rc) return rc;
        Bump b{(uint8_t*)m->scratch, 0, m->scratch_bytes};
        Staged s;
        if ((rc = stage_frame(m, current, b, s))) return rc;
        GridDev g;
        if ((rc = build_grid(m, current, s, b, g))) return rc;
        const orbgpu_keypoint* d_kk = kf_keypoints;
        const orbgpu_mappoint_geometry* d_mps = mappoints;
        const uint8_t* d_mpd = mp_descriptors;
        const uint8_t* d_use = usable;
        const uint8_t* d_claimed = claimed;
        int* d_match = match_out;
        if (mem != ORBGPU_MEM_DEVICE) {
            orbgpu_keypoint* k = b.take<orbgpu_keypoint>(std::max(1, M));
            orbgpu_mappoint_geometry* a = b.take<orbgpu_mappoint_geometry>(std::max(1, M));
            uint8_t* dd = b.take<uint8_t>((size_t)std::max(1, M) * 32);
            uint8_t* uu = b.take<uint8_t>(std::max(1, M));
            if (M) {
                if (kf_keypoints)
                    ORBGPU_CUDA_TRY(cudaMemcpyAsync(k, kf_keypoints, sizeof(orbgpu_keypoint) * M,
                                                    cudaMemcpyHostToDevice, m->stream));
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(a, mappoints, sizeof(orbgpu_mappoint_geometry) * M,
                                                cudaMemcpyHostToDevice, m->stream));
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(dd, mp_descriptors, 32 * (size_t)M, cudaMemcpyHostToDevice,
                                                m->stream));
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(uu, usable, M, cudaMemcpyHostToDevice, m->stream));
            }
            d_kk = k;
            d_mps = a;
            d_mpd = dd;
            d_use = uu;
            if (claimed) {
                uint8_t* c = b.take<uint8_t>(std::max(1, n));
                if (n) ORBGPU_CUDA_TRY(cudaMemcpyAsync(c, claimed, n, cudaMemcpyHostToDevice, m->stream));
                d_claimed = c;
            }
            d_match = b.take<int>(std::max(1, n));
        }
        if (n > 0) k_init_match_out<<<(n + 255) / 256, 256, 0, m->stream>>>(d_claimed, n, d_match);
        int *start, *count, total = 0;
        uint64_t* keys = nullptr;
        auto launch = [&](const int* st, int* cnt, uint64_t* out, int fill) {
            const int wpb = 8;
            if (M > 0)
                k_pkf_candidates<<<(M + wpb - 1) / wpb, 32 * wpb, 0, m->stream>>>(g, kp, d_mps, d_use, d_mpd, M, th,
                                                                               st, cnt, out, fill);
        };
        rc = candidate_lists(m, M, b, launch, start, count, keys, total);
        if (rc == ORBGPU_ERR_CAPACITY) {
            est = est + sizeof(uint64_t) * (size_t)total * 2;
            continue;
        }
        if (rc) return rc;
        int* d_nm = b.take<int>(1);
        int* claims3 = b.take<int>((size_t)3 * std::max(1, n));
        int* res = b.take<int>(std::max(1, M));
        int* changed = b.take<int>(PROJ_ROUNDS);
        int* owner = b.take<int>(std::max(1, n));
        int* nulled = b.take<int>(std::max(1, n));
        int* bin_of = b.take<int>(std::max(1, M));
        ORBGPU_CUDA_TRY(cudaMemsetAsync(d_nm, 0, sizeof(int), m->stream));
        ORBGPU_CUDA_TRY(cudaMemsetAsync(claims3, 0x7f, sizeof(int) * (size_t)3 * std::max(1, n), m->stream));
        ORBGPU_CUDA_TRY(cudaMemsetAsync(res, 0xfe, sizeof(int) * std::max(1, M), m->stream));
        ORBGPU_CUDA_TRY(cudaMemsetAsync(changed, 0, sizeof(int) * PROJ_ROUNDS, m->stream));
        if (M > 0 && n > 0) {
            const int wpb = 8;
            const int warps = std::max(M, (n + 31) / 32);
            // every assignment blocks (src/ORBmatcher.cc:1951: any map point on the keypoint)
            for (int r = 0; r < PROJ_ROUNDS; r++)
                k_pf_round<<<(warps + wpb - 1) / wpb, 32 * wpb, 0, m->stream>>>(n, M, start, count, keys, nullptr, r,
                                                                              claims3, res, changed, d_match);
            k_pf_serial<<<1, 32, 0, m->stream>>>(n, M, start, count, keys, nullptr, changed, res, claims3, d_match);
            // the loop-closing search has no rotation check
            k_pf_finish<<<1, 1024, 0, m->stream>>>(n, M, res, d_kk, s.kps, kp.sim3 ? 0 : m->check_ori, owner, bin_of,
                                                   nulled, d_match, d_nm);
        }
        ORBGPU_CUDA_TRY(cudaGetLastError());
        if (mem != ORBGPU_MEM_DEVICE && n > 0)
            ORBGPU_CUDA_TRY(cudaMemcpyAsync(match_out, d_match, sizeof(int) * n, cudaMemcpyDeviceToHost, m->stream));
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(m->h_pinned, d_nm, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
        ORBGPU_CUDA_TRY(cudaStreamSynchronize(m->stream));
        *nmatches = m->h_pinned[0];
        return ORBGPU_OK;
    }
    return ORBGPU_ERR_CAPACITY;
}

extern "C" int orbgpu_search_by_projection_sim3(orbgpu_matcher* m, const orbgpu_frame* keyframe, const float* Scw,
                                                float fx, float fy, float cx, float cy, float scale_factor,
                                                int nlevels, const orbgpu_mappoint_geometry* points,
                                                const uint8_t* point_descriptors, const uint8_t* usable, int npoints,
                                                int th, const uint8_t* matched, int* match_out, int mem,
                                                int* nmatches) {
    if (!m || !frame_ok(keyframe) || !Scw || npoints < 0 || npoints >= (1 << 20) || !match_out || !nmatches ||
        (npoints > 0 && (!points || !point_descriptors || !usable)) || nlevels < 1 || nlevels > 16 ||
        !(scale_factor > 1.0f))
        return ORBGPU_ERR_BAD_ARG;
    // Scw = [s R | s t]: s = sqrt(row 0 . row 0) (a double dot product, the
    // root rounded to float), R and t divided by it as floats, Ow = -R^T t
    // (src/ORBmatcher.cc:436-442)
    double d = 0.0;
    for (int k = 0; k < 3; k++) d += (double)Scw[k] * (double)Scw[k];
    const float scw = (float)std::sqrt(d);
    KeyframeProjDev kp;
    std::memset(&kp, 0, sizeof(kp));
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 4; c++) kp.T[4 * r + c] = Scw[4 * r + c] / scw;
    for (int i = 0; i < 3; i++) {
        double s = 0.0;
        for (int k = 0; k < 3; k++) s += (double)(-kp.T[4 * k + i]) * (double)kp.T[4 * k + 3];
        kp.Ow[i] = (float)s;
    }
    kp.fx = fx;
    kp.fy = fy;
    kp.cx = cx;
    kp.cy = cy;
    kp.maxX = (float)keyframe->width;
    kp.maxY = (float)keyframe->height;
    // MapPoint::PredictScale(dist, KeyFrame*): the thresholds of the frame version
    orbgpu_frustum_frame tmp;
    const float eye[12] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0};
    int rc = orbgpu_frustum_frame_init(eye, fx, fy, cx, cy, 0, 0, 1, 0, 1, scale_factor, nlevels, &tmp);
    if (rc) return rc;
    kp.nlevels = nlevels;
    std::memcpy(kp.level_above, tmp.level_above, sizeof(kp.level_above));
    kp.orbdist = ORBGPU_TH_LOW;
    kp.sim3 = 1;
    return search_projection_keyframe(m, keyframe, kp, nullptr, points, point_descriptors, usable, npoints, (float)th,
                                      matched, match_out, mem, nmatches);
}

// Fuse's choice per map point: the first least distance of its candidates
// (candidates are already cut at TH_LOW), with no interaction between map
// points -- the map updates it leads to are applied in order by the caller.
__global__ void k_fuse_pick(int m, const int* cand_start, const int* cand_count, const uint64_t* cands,
                            int* target, int* dist_out) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i >= m) return;
    uint64_t best = ~0ull;
    for (int b = lane; b < cand_count[i]; b += 32) {
        const uint64_t key = cands[cand_start[i] + b];
        best = key < best ? key : best;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t ob = __shfl_xor_sync(0xffffffffu, best, o);
        best = ob < best ? ob : best;
    }
    if (lane == 0) {
        target[i] = best == ~0ull ? -1 : (int)(best & 0xFFFFF);
        if (dist_out) dist_out[i] = best == ~0ull ? 256 : (int)(best >> 40);
    }
}

static int fuse_pick_run(orbgpu_matcher* m, const orbgpu_frame* keyframe, const KeyframeProjDev& kp,
                         const orbgpu_mappoint_geometry* mappoints, const uint8_t* mp_descriptors,
                         const uint8_t* usable, int n_mp, float th, int* target, int* dist, int mem);

extern "C" int orbgpu_fuse_candidates(orbgpu_matcher* m, const orbgpu_frame* keyframe, const float* Tcw, float fx,
                                      float fy, float cx, float cy, float bf, float scale_factor, int nlevels,
                                      const float* inv_level_sigma2, const orbgpu_mappoint_geometry* mappoints,
                                      const uint8_t* mp_descriptors, const uint8_t* usable, int n_mp, float th,
                                      int* target, int* dist, int mem) {
    if (!m || !frame_ok(keyframe) || !Tcw || !inv_level_sigma2 || n_mp < 0 || n_mp >= (1 << 20) || !target ||
        (n_mp > 0 && (!mappoints || !mp_descriptors || !usable)) || nlevels < 1 || nlevels > 16 ||
        !(scale_factor > 1.0f))
        return ORBGPU_ERR_BAD_ARG;
    KeyframeProjDev kp;
    std::memset(&kp, 0, sizeof(kp));
    std::memcpy(kp.T, Tcw, sizeof(kp.T));
    // Ow = GetCameraCenter() = -Rcw^T tcw
    for (int i = 0; i < 3; i++) {
        double s = 0.0;
        for (int k = 0; k < 3; k++) s += (double)(-Tcw[4 * k + i]) * (double)Tcw[4 * k + 3];
        kp.Ow[i] = (float)s;
    }
    kp.fx = fx;
    kp.fy = fy;
    kp.cx = cx;
    kp.cy = cy;
    kp.bf = bf;
    kp.maxX = (float)keyframe->width;
    kp.maxY = (float)keyframe->height;
    orbgpu_frustum_frame tmp;
    const float eye[12] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0};
    int rc = orbgpu_frustum_frame_init(eye, fx, fy, cx, cy, 0, 0, 1, 0, 1, scale_factor, nlevels, &tmp);
    if (rc) return rc;
    kp.nlevels = nlevels;
    std::memcpy(kp.level_above, tmp.level_above, sizeof(kp.level_above));
    for (int l = 0; l < nlevels; l++) kp.inv_sigma2[l] = inv_level_sigma2[l];
    kp.orbdist = ORBGPU_TH_LOW;
    kp.sim3 = 1;
    kp.fuse = 1;
    return fuse_pick_run(m, keyframe, kp, mappoints, mp_descriptors, usable, n_mp, th, target, dist, mem);
}

// The candidate lists of a fuse search and the choice of every map point.
static int fuse_pick_run(orbgpu_matcher* m, const orbgpu_frame* keyframe, const KeyframeProjDev& kp,
                         const orbgpu_mappoint_geometry* mappoints, const uint8_t* mp_descriptors,
                         const uint8_t* usable, int n_mp, float th, int* target, int* dist, int mem) {
    int rc;
    const int n = keyframe->n, M = n_mp;
    size_t est = frame_stage_bytes(keyframe) + grid_bytes(n) +
                 (size_t)std::max(1, M) * (sizeof(orbgpu_mappoint_geometry) + 32 + 1 + 2 * sizeof(int) + 32) +
                 64 * 1024 + sizeof(uint64_t) * (size_t)std::max(1, M) * 32;
    for (int attempt = 0; attempt < 2; attempt++) {
        rc = ensure_scratch(m, est);
        if (rc) return rc;
        Bump b{(uint8_t*)m->scratch, 0, m->scratch_bytes};
        Staged s;
        if ((rc = stage_frame(m, keyframe, b, s))) return rc;
        GridDev g;
        if ((rc = build_grid(m, keyframe, s, b, g))) return rc;
        const orbgpu_mappoint_geometry* d_mps = mappoints;
        const uint8_t* d_mpd = mp_descriptors;
        const uint8_t* d_use = usable;
        int* d_t = target;
        int* d_d = dist;
        if (mem != ORBGPU_MEM_DEVICE) {
            orbgpu_mappoint_geometry* a = b.take<orbgpu_mappoint_geometry>(std::max(1, M));
            uint8_t* dd = b.take<uint8_t>((size_t)std::max(1, M) * 32);
            uint8_t* uu = b.take<uint8_t>(std::max(1, M));
            if (M) {
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(a, mappoints, sizeof(orbgpu_mappoint_geometry) * M,
                                                cudaMemcpyHostToDevice, m->stream));
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(dd, mp_descriptors, 32 * (size_t)M, cudaMemcpyHostToDevice,
                                                m->stream));
                ORBGPU_CUDA_TRY(cudaMemcpyAsync(uu, usable, M, cudaMemcpyHostToDevice, m->stream));
            }
            d_mps = a;
            d_mpd = dd;
            d_use = uu;
            d_t = b.take<int>(std::max(1, M));
            d_d = dist ? b.take<int>(std::max(1, M)) : nullptr;
        }
        int *start, *count, total = 0;
        uint64_t* keys = nullptr;
        auto launch = [&](const int* st, int* cnt, uint64_t* out, int fill) {
            const int wpb = 8;
            if (M > 0)
                k_pkf_candidates<<<(M + wpb - 1) / wpb, 32 * wpb, 0, m->stream>>>(g, kp, d_mps, d_use, d_mpd, M, th,
                                                                               st, cnt, out, fill);
        };
        rc = candidate_lists(m, M, b, launch, start, count, keys, total);
        if (rc == ORBGPU_ERR_CAPACITY) {
            est = est + sizeof(uint64_t) * (size_t)total * 2;
            continue;
        }
        if (rc) return rc;
        if (M > 0) k_fuse_pick<<<(M + 7) / 8, 256, 0, m->stream>>>(M, start, count, keys, d_t, d_d);
        ORBGPU_CUDA_TRY(cudaGetLastError());
        if (mem != ORBGPU_MEM_DEVICE && M > 0) {
            ORBGPU_CUDA_TRY(cudaMemcpyAsync(target, d_t, sizeof(int) * M, cudaMemcpyDeviceToHost, m->stream));
            if (dist) ORBGPU_CUDA_TRY(cudaMemcpyAsync(dist, d_d, sizeof(int) * M, cudaMemcpyDeviceToHost, m->stream));
        }
        ORBGPU_CUDA_TRY(cudaStreamSynchronize(m->stream));
        return ORBGPU_OK;
    }
    return ORBGPU_ERR_CAPACITY;
}

extern "C" int orbgpu_fuse_sim3_candidates(orbgpu_matcher* m, const orbgpu_frame* keyframe, const float* Scw,
                                           float fx, float fy, float cx, float cy, float scale_factor, int nlevels,
                                           const orbgpu_mappoint_geometry* points, const uint8_t* point_descriptors,
                                           const uint8_t* usable, int npoints, float th, int* target, int* dist,
                                           int mem) {
    if (!m || !frame_ok(keyframe) || !Scw || npoints < 0 || npoints >= (1 << 20) || !target ||
        (npoints > 0 && (!points || !point_descriptors || !usable)) || nlevels < 1 || nlevels > 16 ||
        !(scale_factor > 1.0f))
        return ORBGPU_ERR_BAD_ARG;
    // the Sim3 de-scaled as in SearchByProjection(KeyFrame*, Scw, ...)
    double d = 0.0;
    for (int k = 0; k < 3; k++) d += (double)Scw[k] * (double)Scw[k];
    const float scw = (float)std::sqrt(d);
    KeyframeProjDev kp;
    std::memset(&kp, 0, sizeof(kp));
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 4; c++) kp.T[4 * r + c] = Scw[4 * r + c] / scw;
    for (int i = 0; i < 3; i++) {
        double s = 0.0;
        for (int k = 0; k < 3; k++) s += (double)(-kp.T[4 * k + i]) * (double)kp.T[4 * k + 3];
        kp.Ow[i] = (float)s;
    }
    kp.fx = fx;
    kp.fy = fy;
    kp.cx = cx;
    kp.cy = cy;
    kp.maxX = (float)keyframe->width;
    kp.maxY = (float)keyframe->height;
    orbgpu_frustum_frame tmp;
    const float eye[12] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0};
    int rc = orbgpu_frustum_frame_init(eye, fx, fy, cx, cy, 0, 0, 1, 0, 1, scale_factor, nlevels, &tmp);
    if (rc) return rc;
    kp.nlevels = nlevels;
    std::memcpy(kp.level_above, tmp.level_above, sizeof(kp.level_above));
    kp.orbdist = ORBGPU_TH_LOW;
    kp.sim3 = 1;
    kp.invz_double = 1;
    return fuse_pick_run(m, keyframe, kp, points, point_descriptors, usable, npoints, th, target, dist, mem);
}

// SearchBySim3's geometry: cv::Mat products accumulated in double and
// rounded to float (plus a float add), scalar products of float matrices as
// float products of the scalar rounded to float.
static void mat3_times(const float* A, const float* x, float* out) {
    for (int r = 0; r < 3; r++) {
        double s = 0.0;
        for (int k = 0; k < 3; k++) s += (double)A[3 * r + k] * (double)x[k];
        out[r] = (float)s;
    }
}

extern "C" int orbgpu_search_by_sim3(orbgpu_matcher* m, const orbgpu_frame* kf1, const orbgpu_frame* kf2,
                                     const float* T1w, const float* T2w, float s12, const float* R12,
                                     const float* t12, float fx, float fy, float cx, float cy, float scale_factor,
                                     int nlevels, const orbgpu_mappoint_geometry* mps1, const uint8_t* mpd1,
                                     const uint8_t* usable1, const orbgpu_mappoint_geometry* mps2,
                                     const uint8_t* mpd2, const uint8_t* usable2, float th, int* match12,
                                     int* nfound) {
    if (!m || !frame_ok(kf1) || !frame_ok(kf2) || !T1w || !T2w || !R12 || !t12 || !match12 || !nfound ||
        nlevels < 1 || nlevels > 16 || !(scale_factor > 1.0f) || kf1->n < 0 || kf2->n < 0 ||
        (kf1->n > 0 && (!mps1 || !mpd1 || !usable1)) || (kf2->n > 0 && (!mps2 || !mpd2 || !usable2)))
        return ORBGPU_ERR_BAD_ARG;
    const int N1 = kf1->n, N2 = kf2->n;
    // sR12 = s12 * R12, sR21 = (1.0 / s12) * R12^T, t21 = -sR21 * t12
    // (src/ORBmatcher.cc:1456-1463)
    const float inv_s = (float)(1.0 / (double)s12);
    float sR12[9], sR21[9], nsR21[9], t21[3];
    for (int r = 0; r < 3; r++)
        for (int c = 0; c < 3; c++) {
            sR12[3 * r + c] = R12[3 * r + c] * s12;
            sR21[3 * r + c] = R12[3 * c + r] * inv_s;
            nsR21[3 * r + c] = -sR21[3 * r + c];
        }
    mat3_times(nsR21, t12, t21);
    orbgpu_frustum_frame tmp;
    const float eye[12] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0};
    int rc = orbgpu_frustum_frame_init(eye, fx, fy, cx, cy, 0, 0, 1, 0, 1, scale_factor, nlevels, &tmp);
    if (rc) return rc;
    auto pass = [&](const orbgpu_frame* target_kf, const float* Tw, const float* sR, const float* t,
                    const orbgpu_mappoint_geometry* mps, const uint8_t* mpd, const uint8_t* use, int n,
                    std::vector<int>& out) {
        KeyframeProjDev kp;
        std::memset(&kp, 0, sizeof(kp));
        std::memcpy(kp.T, Tw, sizeof(kp.T));
        for (int r = 0; r < 3; r++) {
            for (int c = 0; c < 3; c++) kp.T2[4 * r + c] = sR[3 * r + c];
            kp.T2[4 * r + 3] = t[r];
        }
        kp.fx = fx;
        kp.fy = fy;
        kp.cx = cx;
        kp.cy = cy;
        kp.maxX = (float)target_kf->width;
        kp.maxY = (float)target_kf->height;
        kp.nlevels = nlevels;
        std::memcpy(kp.level_above, tmp.level_above, sizeof(kp.level_above));
        kp.orbdist = ORBGPU_TH_HIGH;
        kp.sim3 = 1;
        kp.invz_double = 1;
        kp.chain = 1;
        out.assign(std::max(n, 1), -1);
        return fuse_pick_run(m, target_kf, kp, mps, mpd, use, n, th, out.data(), nullptr, ORBGPU_MEM_HOST);
    };
    // vnMatch1: pKF1's map points into pKF2; vnMatch2: pKF2's into pKF1
    std::vector<int> match1, match2;
    if ((rc = pass(kf2, T1w, sR21, t21, mps1, mpd1, usable1, N1, match1))) return rc;
    if ((rc = pass(kf1, T2w, sR12, t12, mps2, mpd2, usable2, N2, match2))) return rc;
    int found = 0;
    for (int i1 = 0; i1 < N1; i1++) {
        const int i2 = match1[i1];
        match12[i1] = (i2 >= 0 && i2 < N2 && match2[i2] == i1) ? i2 : -1;
        found += match12[i1] >= 0;
    }
    *nfound = found;
    return ORBGPU_OK;
}

extern "C" int orbgpu_compute_stereo_matches(orbgpu_matcher* m, const orbgpu_extractor* left,
                                             const orbgpu_extractor* right, const orbgpu_frame* fl,
                                             const orbgpu_frame* fr, float bf, float fx, float* uright, float* depth,
                                             int mem) {
    if (!m || !left || !right || !frame_ok(fl) || !frame_ok(fr) || !uright || !depth) return ORBGPU_ERR_BAD_ARG;
    const int nL = fl->n, nR = fr->n;
    if (nL == 0) return ORBGPU_OK;
    StereoLevels lv;
    std::memset(&lv, 0, sizeof(lv));
    int nlev = fl->nlevels;
    for (int l = 0; l < nlev; l++) {
        const uint8_t *pl, *pr;
        int w, h, w2, h2;
        size_t pitch, pitch2;
        if (orbgpu_extractor_pyramid_level(left, l, &pl, &w, &h, &pitch) ||
            orbgpu_extractor_pyramid_level(right, l, &pr, &w2, &h2, &pitch2) || w != w2 || h != h2 || pitch != pitch2)
            return ORBGPU_ERR_BAD_ARG;
        lv.left[l] = pl;
        lv.right[l] = pr;
        lv.w[l] = w;
        lv.h[l] = h;
        lv.pitch[l] = (int)pitch;
        lv.scale[l] = fl->scale_factors[l];
        lv.inv_scale[l] = 1.0f / fl->scale_factors[l];
    }
    lv.nlevels = nlev;
    const int nRows = lv.h[0];
    const size_t est = frame_stage_bytes(fl) + frame_stage_bytes(fr) + (ORBGPU_MAX_DIM + 1) * sizeof(int) +
                       (size_t)nR * sizeof(uint4) + (size_t)nL * 3 * sizeof(float) + 64 * 1024;
    int rc = ensure_scratch(m, est);
    if (rc) return rc;
    Bump b{(uint8_t*)m->scratch, 0, m->scratch_bytes};
    Staged sl, sr;
    if ((rc = stage_frame(m, fl, b, sl)) || (rc = stage_frame(m, fr, b, sr))) return rc;
    int* row_start = b.take<int>(ORBGPU_MAX_DIM + 1);
    uint4* recs = b.take<uint4>(std::max(1, nR));
    float* d_ur = uright;
    float* d_dp = depth;
    if (mem != ORBGPU_MEM_DEVICE) {
        d_ur = b.take<float>(nL);
        d_dp = b.take<float>(nL);
    }
    int* sad = b.take<int>(nL);
    int* status = b.take<int>(1);
    k_stereo_index<<<1, STEREO_INDEX_THREADS, 0, m->stream>>>(sr.kps, nR, nlev, nRows, row_start, recs, status);
    k_stereo_match<<<(nL + STEREO_WARPS - 1) / STEREO_WARPS, 32 * STEREO_WARPS, 0, m->stream>>>(
        sl.kps, sl.desc, nL, sr.desc, lv, nRows, row_start, recs, bf, fx, d_ur, d_dp, sad, status);
    k_stereo_median<<<1, STEREO_INDEX_THREADS, 0, m->stream>>>(nL, sad, d_ur, d_dp);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    if (mem != ORBGPU_MEM_DEVICE) {
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(uright, d_ur, sizeof(float) * nL, cudaMemcpyDeviceToHost, m->stream));
        ORBGPU_CUDA_TRY(cudaMemcpyAsync(depth, d_dp, sizeof(float) * nL, cudaMemcpyDeviceToHost, m->stream));
    }
    ORBGPU_CUDA_TRY(cudaMemcpyAsync(m->h_pinned, status, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    ORBGPU_CUDA_TRY(cudaStreamSynchronize(m->stream));
    if (m->h_pinned[0]) {
        orbgpu_set_last_error("stereo patch outside its level", __FILE__, __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    return ORBGPU_OK;
}

extern "C" int orbgpu_descriptor_distance(const uint8_t* a, const uint8_t* b, int n, int* out, void* stream) {
    if (n < 0 || (n > 0 && (!a || !b || !out))) return ORBGPU_ERR_BAD_ARG;
    if (n == 0) return ORBGPU_OK;
    k_descriptor_distance<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(a, b, n, out);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    return ORBGPU_OK;
}

// ---------------------------------------------------------------- internal access for the kNN file
cudaStream_t orbgpu_matcher_stream_internal(orbgpu_matcher* m) { return m->stream; }
