// orbgpu_grid.cuh -- Frame's 64 x 48 keypoint grid (AssignFeaturesToGrid,
// src/Frame.cc:399-423), the walk over a search window's cells
// (GetFeaturesInArea, src/Frame.cc:590-670) and the parts of
// SearchByProjection (src/ORBmatcher.cc:72-183) that the per-frame and the
// batched searches share.
#pragma once

#include "orbgpu_common.cuh"

namespace orbgpu {

#define ORBGPU_GRID_CELLS (ORBGPU_GRID_COLS * ORBGPU_GRID_ROWS)

// A keypoint as the window walks read it, in cell order: one 16-byte load
// gives what three dependent ones did (the cell's key list, the key's cell
// and the 28-byte keypoint).
struct __align__(16) GridRec {
    float x, y;
    uint32_t cell_oct;  // cell (ix * 48 + iy) | octave << 24, the octave clamped to a signed byte
    uint32_t idx;
    __device__ __forceinline__ int cell() const { return (int)(cell_oct & 0xFFFFFFu); }
    __device__ __forceinline__ int octave() const { return (int)cell_oct >> 24; }
};

// PosInGrid (src/Frame.cc:682-698); -1 outside the grid.
__device__ __forceinline__ int pos_in_grid(const orbgpu_keypoint& kp, float minX, float minY, float invW, float invH) {
    const int px = (int)roundf(__fmul_rn(__fsub_rn(kp.x, minX), invW));
    const int py = (int)roundf(__fmul_rn(__fsub_rn(kp.y, minY), invH));
    if (px < 0 || px >= ORBGPU_GRID_COLS || py < 0 || py >= ORBGPU_GRID_ROWS) return -1;
    return px * ORBGPU_GRID_ROWS + py;
}

__device__ __forceinline__ GridRec grid_rec(const orbgpu_keypoint& kp, int cell, int i) {
    GridRec r;
    r.x = kp.x;
    r.y = kp.y;
    r.cell_oct = (uint32_t)cell | ((uint32_t)min(max(kp.octave, -128), 127) << 24);
    r.idx = (uint32_t)i;
    return r;
}

// One frame's cell starts by one block of 1024 threads: counts in shared
// memory (s_cell) and their exclusive scan, three consecutive cells per
// thread.  Leaves the starts in s_cell too, as the cells' fill positions.
__device__ __forceinline__ void grid_starts_block(const orbgpu_keypoint* kps, int n, float minX, float minY, float invW,
                                                  float invH, int (&s_cell)[ORBGPU_GRID_CELLS], int* cell_start) {
    constexpr int PER = ORBGPU_GRID_CELLS / 1024;
    static_assert(ORBGPU_GRID_CELLS % 1024 == 0, "whole cells per thread");
    __shared__ int s_scan[32];
    const int t = threadIdx.x;
    for (int c = t; c < ORBGPU_GRID_CELLS; c += 1024) s_cell[c] = 0;
    __syncthreads();
    for (int i = t; i < n; i += 1024) {
        const int c = pos_in_grid(kps[i], minX, minY, invW, invH);
        if (c >= 0) atomicAdd(&s_cell[c], 1);
    }
    __syncthreads();
    int v[PER], sum = 0;
#pragma unroll
    for (int k = 0; k < PER; k++) {
        v[k] = s_cell[PER * t + k];
        sum += v[k];
    }
    int total;
    int at = block_exclusive_scan(sum, s_scan, &total);
#pragma unroll
    for (int k = 0; k < PER; k++) {
        cell_start[PER * t + k] = at;
        s_cell[PER * t + k] = at;
        at += v[k];
    }
    if (t == 0) cell_start[ORBGPU_GRID_CELLS] = total;
    __syncthreads();
}

// The starts, then the records into their cells (the order inside a cell does
// not matter: searches compare (distance, cell, index)).
__device__ __forceinline__ void grid_build_block(const orbgpu_keypoint* kps, int n, float minX, float minY, float invW,
                                                 float invH, int* cell_start, GridRec* recs) {
    __shared__ int s_cell[ORBGPU_GRID_CELLS];
    grid_starts_block(kps, n, minX, minY, invW, invH, s_cell, cell_start);
    for (int i = threadIdx.x; i < n; i += 1024) {
        const orbgpu_keypoint kp = kps[i];
        const int c = pos_in_grid(kp, minX, minY, invW, invH);
        if (c >= 0) recs[atomicAdd(&s_cell[c], 1)] = grid_rec(kp, c, i);
    }
}

// The grid records of the cells [x0, x1] x [y0, y1] for W-lane segments of a
// warp (W = 8, 16 or 32), each segment with its own window: segment g holds
// lanes [g W, g W + W).  Cells are stored column-major (cell = x * rows + y)
// and their records back to back, so the window's records of grid column x
// are one range: one lane per column instead of one per cell.  Records are
// visited column by column, cell by cell within a column, as
// GetFeaturesInArea visits the keypoints.  Every lane of the warp runs the
// loops to the longest segment's bounds (a segment with active == false, or
// past its own bounds, visits with valid == false and a record of zeros), so
// the visitor may use full-warp ballots and shuffles.
template <int W, typename Visit>
__device__ __forceinline__ void seg_window_recs(const int* cell_start, const GridRec* recs, bool active, int x0, int x1,
                                                int y0, int y1, Visit visit) {
    static_assert(W == 8 || W == 16 || W == 32, "segment width");
    const int sl = (threadIdx.x & 31) & (W - 1);
    const int ncol = active && y1 >= y0 ? x1 - x0 + 1 : 0;
    int nmax = ncol;
#pragma unroll
    for (int o = W; o < 32; o <<= 1) nmax = max(nmax, __shfl_xor_sync(0xffffffffu, nmax, o));
    for (int c0 = 0; c0 < nmax; c0 += W) {
        const int cx = c0 + sl;
        int s = 0, n = 0;
        if (cx < ncol) {
            const int base = (x0 + cx) * ORBGPU_GRID_ROWS;
            s = cell_start[base + y0];
            n = cell_start[base + y1 + 1] - s;
        }
        int incl = n;
#pragma unroll
        for (int o = 1; o < W; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o, W);
            if (sl >= o) incl += y;
        }
        const int total = __shfl_sync(0xffffffffu, incl, W - 1, W);
        const int excl = incl - n;
        int tmax = total;
#pragma unroll
        for (int o = W; o < 32; o <<= 1) tmax = max(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
        for (int t0 = 0; t0 < tmax; t0 += W) {
            const int t = t0 + sl;
            // the last lane of the segment whose range starts at or before t holds entry t
            int k = 0;
#pragma unroll
            for (int step = W / 2; step > 0; step >>= 1) {
                const int e = __shfl_sync(0xffffffffu, excl, k + step, W);
                if (e <= t) k += step;
            }
            const int sk = __shfl_sync(0xffffffffu, s, k, W);
            const int ek = __shfl_sync(0xffffffffu, excl, k, W);
            const bool valid = t < total;
            GridRec r{0.f, 0.f, 0u, 0u};
            if (valid) r = recs[sk + t - ek];
            visit(r, valid);
        }
    }
}

// Frame::GetFeaturesInArea's disc.
__device__ __forceinline__ bool in_disc(const GridRec& r, float x, float y, float rr) {
    const float dx = __fsub_rn(r.x, x), dy = __fsub_rn(r.y, y);
    return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)) < rr;
}

// Candidate keys in the order of GetFeaturesInArea ("first strictly smaller
// wins" is the least (distance, cell, index)): 32 bits for distances below
// 256 and indices below 4096, 64 bits for all.
template <typename Key>
__device__ __forceinline__ Key make_key(int dist, int cell, int idx);
template <>
__device__ __forceinline__ uint32_t make_key<uint32_t>(int dist, int cell, int idx) {
    return ((uint32_t)dist << 24) | ((uint32_t)cell << 12) | (uint32_t)idx;
}
template <>
__device__ __forceinline__ uint64_t make_key<uint64_t>(int dist, int cell, int idx) {
    return ((uint64_t)(uint32_t)dist << 40) | ((uint64_t)(uint32_t)cell << 20) | (uint64_t)(uint32_t)idx;
}
#define ORBGPU_KEY32_MAX_N 4096  // keypoints with 32-bit keys

// One frame as SearchByProjection's candidates read it.
struct ProjFrame {
    const int* cell_start;
    const GridRec* recs;
    const uint8_t* desc;
    const float* uright;  // or null
    float minX, minY, invW, invH;
    const float* scale;  // 16
};

// The candidates of one map point per W-lane segment of the warp
// (src/ORBmatcher.cc:84-145): keypoints in the scaled window over levels
// [L - 1, L] that pass the stereo gate, with their distances, into
// row[0, slot_cap); returns how many there are.  A candidate with nnratio *
// dist > TH_HIGH (nnratio <= 1) can neither be accepted (dist > TH_HIGH) nor
// make an accepted best fail the ratio test (best <= TH_HIGH < nnratio *
// dist), and one at 256 is never below the reference's initial best: the
// lists leave them out.
template <int W, typename Key>
__device__ __forceinline__ int proj_candidates(const ProjFrame& F, const orbgpu_mappoint& mp, bool have,
                                               const uint8_t* mp_desc, float th, float nnratio, Key* row, int slot_cap) {
    const bool drop_far = nnratio <= 1.0f;
    const int lane = threadIdx.x & 31, sbase = lane & ~(W - 1);
    const unsigned smask = (W == 32 ? 0xffffffffu : ((1u << (W & 31)) - 1)) << sbase;
    bool active = have && mp.track_in_view && !mp.bad && mp.track_scale_level >= 0 && mp.track_scale_level < 16;
    int x0 = 0, x1 = -1, y0 = 0, y1 = -1, level = 0;
    float x = 0.f, y = 0.f, rr = 0.f, radius = 0.f;
    uint4 dm0 = make_uint4(0, 0, 0, 0), dm1 = dm0;  // the map point's descriptor
    if (active) {
        level = mp.track_scale_level;
        float r = mp.view_cos > 0.998f ? 2.5f : 4.0f;  // RadiusByViewingCos, src/ORBmatcher.cc:186-193
        if (th != 1.0f) r = __fmul_rn(r, th);
        radius = __fmul_rn(r, F.scale[level]);
        x = mp.proj_x;
        y = mp.proj_y;
        x0 = max(0, (int)floorf(__fmul_rn(__fsub_rn(__fsub_rn(x, F.minX), radius), F.invW)));
        x1 = min(ORBGPU_GRID_COLS - 1, (int)ceilf(__fmul_rn(__fadd_rn(__fsub_rn(x, F.minX), radius), F.invW)));
        y0 = max(0, (int)floorf(__fmul_rn(__fsub_rn(__fsub_rn(y, F.minY), radius), F.invH)));
        y1 = min(ORBGPU_GRID_ROWS - 1, (int)ceilf(__fmul_rn(__fadd_rn(__fsub_rn(y, F.minY), radius), F.invH)));
        active = x0 < ORBGPU_GRID_COLS && x1 >= 0 && y0 < ORBGPU_GRID_ROWS && y1 >= 0 && x0 <= x1 && y0 <= y1;
        rr = __fmul_rn(radius, radius);
    }
    if (active) {
        const uint4* dp = reinterpret_cast<const uint4*>(mp_desc);
        dm0 = dp[0];
        dm1 = dp[1];
    }
    int total = 0;
    seg_window_recs<W>(F.cell_start, F.recs, active, x0, x1, y0, y1, [&](const GridRec& rec, bool valid) {
        bool ok = valid && rec.octave() >= level - 1 && rec.octave() <= level && in_disc(rec, x, y, rr);
        if (ok && F.uright) {
            const float ur = F.uright[rec.idx];
            if (ur > 0) ok = !(fabsf(__fsub_rn(mp.proj_xr, ur)) > radius);
        }
        int dist = 256;
        if (ok) {
            const uint4* kd = reinterpret_cast<const uint4*>(F.desc + (size_t)rec.idx * 32);
            dist = hamming256(dm0, dm1, kd[0], kd[1]);
            ok = dist < 256 && !(drop_far && __fmul_rn(nnratio, (float)dist) > (float)ORBGPU_TH_HIGH);
        }
        const unsigned msk = __ballot_sync(0xffffffffu, ok) & smask;
        if (ok) {
            const int pos = total + __popc(msk & ((1u << lane) - 1));
            if (pos < slot_cap) row[pos] = make_key<Key>(dist, rec.cell(), (int)rec.idx);
        }
        total += __popc(msk);
    });
    return total;
}

#define PROJ_NOKEY 0xFFFFFFFFu
#define PROJ_FREE 0x7fffffff
// Inserts a key into the N smallest so far.
template <int N>
__device__ __forceinline__ void top_insert(uint32_t (&t)[N], uint32_t k) {
#pragma unroll
    for (int j = 0; j < N; j++) {
        const uint32_t lo = min(t[j], k);
        k = max(t[j], k);
        t[j] = lo;
    }
}
// Calls visit(key) for the cnt keys of a candidate row (16-byte aligned,
// 32-bit keys), and for up to 7 more PROJ_NOKEY: two 16-byte loads in flight.
template <typename Visit>
__device__ __forceinline__ void row_visit(const uint32_t* row, int cnt, Visit visit) {
    for (int b = 0; b < cnt; b += 8) {
        const uint4 v = reinterpret_cast<const uint4*>(row)[b >> 2];
        uint4 w = make_uint4(PROJ_NOKEY, PROJ_NOKEY, PROJ_NOKEY, PROJ_NOKEY);
        if (b + 4 < cnt) w = reinterpret_cast<const uint4*>(row)[(b >> 2) + 1];
        const uint32_t k[8] = {v.x, v.y, v.z, v.w, w.x, w.y, w.z, w.w};
#pragma unroll
        for (int j = 0; j < 8; j++) visit(b + j < cnt ? k[j] : PROJ_NOKEY);
    }
}
// The N smallest keys of a row.
template <int N>
__device__ __forceinline__ void top_load(const uint32_t* row, int cnt, uint32_t (&t)[N]) {
#pragma unroll
    for (int j = 0; j < N; j++) t[j] = PROJ_NOKEY;
    row_visit(row, cnt, [&](uint32_t k) { top_insert(t, k); });
}

// The in-order resolution of SearchByProjection(Frame&, vector<MapPoint*>)
// for one frame by one block, as a fixed point: in the reference a map point
// sees a keypoint as claimed iff an earlier map point of the call took it.
// Round r evaluates every map point against the claims of round r - 1's
// results (claim owner = smallest map point index that took the keypoint);
// once a round changes no result, every map point's result is consistent with
// those before it, which by induction over the map point order is the
// sequential result (at most M + 1 rounds: round r fixes the first r + 1).
// A map point's result is the first two unclaimed candidates in key order:
// Each thread keeps the four smallest keys of its first PROJ_MPT map points in
// registers and the next four in shared memory (from 'tops', the eight smallest
// of every map point, or its row where that is null).  It looks behind the
// fourth (and behind the eighth, at the whole row) only where that can matter:
// with nothing unclaimed before, while the keys are not above TH_HIGH (no later
// one is accepted); with the best only, while a key could still fail the ratio
// test.  Shared memory: the keys (16 bytes a map point), results of the map
// points past the registers', two claim arrays (4096 ints: index 4095, that of
// PROJ_NOKEY, is never free) and the octaves (n bytes).  'claimed' (or null):
// keypoints taken before the call, reported as -2.
// At M = 3000 on 1000 to 2000 keypoints (lists of 3 to 5 keys, 18 at most, about
// ten rounds) bound by its instructions, about 60 a map point and round: 46 us
// for the 64 frames of the batched step (64 blocks), 19 for one frame; with the
// lists walked to their ends 77, and 12 launches of a round each for one frame.
#define PROJ_MPT 4  // map points per thread with keys in registers
#define PROJ_TOP 8  // keys of a map point outside its row
__host__ __device__ inline size_t proj_resolve_smem(int n, int M) {
    const size_t regs = 1024 * PROJ_MPT, mr = (size_t)M < regs ? (size_t)M : regs;
    return 16 * mr + 4 * ((size_t)M - mr + 2 * ORBGPU_KEY32_MAX_N) + (size_t)n + 16;
}
// Returns the rounds run, 0 when they did not converge.
__device__ __forceinline__ int proj_resolve_block(const orbgpu_keypoint* kps, int n, int M, const uint32_t* slots,
                                                  int slot_cap, const int* slot_count, const uint4* tops, float nnratio,
                                                  const uint8_t* claimed, int* smem, int* match_out, int* nmatches) {
    __shared__ int s_scan[32];
    __shared__ int s_flag[3];
    const int tid = threadIdx.x, nt = blockDim.x;
    const int Mr = min(M, PROJ_MPT * 1024);  // a block of 1024 threads
    uint4* s_next = reinterpret_cast<uint4*>(smem);         // Mr: keys 4 .. 7
    int* s_res = reinterpret_cast<int*>(s_next + Mr) - Mr;  // [Mr, M): results
    int* cr = s_res + M;                                    // claims of the previous round
    int* cw = cr + ORBGPU_KEY32_MAX_N;                      // claims of this round
    uint8_t* s_oct = reinterpret_cast<uint8_t*>(cw + ORBGPU_KEY32_MAX_N);
    if (tid < 3) s_flag[tid] = 0;
    for (int k = tid; k < ORBGPU_KEY32_MAX_N; k += nt) {
        // a keypoint claimed before the call has an owner before every map point
        cr[k] = cw[k] = k >= n || (claimed && claimed[k]) ? -1 : PROJ_FREE;
        if (k < n) s_oct[k] = (uint8_t)kps[k].octave;
    }
    uint32_t top[PROJ_MPT][4];
    int cnt[PROJ_MPT], res[PROJ_MPT];
#pragma unroll
    for (int q = 0; q < PROJ_MPT; q++) {
        const int i = tid + q * nt;
        cnt[q] = i < M ? min(slot_count[i], slot_cap) : 0;
        res[q] = -2;
    }
#pragma unroll
    for (int q = 0; q < PROJ_MPT; q++) {
        const int i = tid + q * nt;
        uint32_t t[PROJ_TOP];
        if (!tops) {
            top_load(slots + (size_t)i * slot_cap, cnt[q], t);
        } else {
#pragma unroll
            for (int l = 0; l < 2; l++) {
                uint4 v = make_uint4(PROJ_NOKEY, PROJ_NOKEY, PROJ_NOKEY, PROJ_NOKEY);
                if (cnt[q] > 4 * l) v = tops[2 * (size_t)i + l];
                t[4 * l] = v.x;
                t[4 * l + 1] = v.y;
                t[4 * l + 2] = v.z;
                t[4 * l + 3] = v.w;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) top[q][j] = t[j];
        if (cnt[q] > 4) s_next[i] = make_uint4(t[4], t[5], t[6], t[7]);
    }
    for (int i = Mr + tid; i < M; i += nt) s_res[i] = -2;
    auto dist_of = [](uint32_t key) { return (int)(key >> 24); };  // 255 for PROJ_NOKEY
    auto ratio_fails = [&](uint32_t best, uint32_t key) {
        return (float)dist_of(best) > __fmul_rn(nnratio, (float)dist_of(key));
    };
    auto decide = [&](uint32_t best, uint32_t second) -> int {
        if (dist_of(best) > ORBGPU_TH_HIGH) return -1;
        const int b = (int)(best & 0xFFFu);
        // no second: bestDist2 256 and a level that equals none
        if (second != PROJ_NOKEY && ratio_fails(best, second) && s_oct[b] == s_oct[second & 0xFFFu]) return -1;
        return b;
    };
    // the first two unclaimed of four keys in order, after (best, second)
    auto pick = [&](int i, const uint32_t (&t)[4], uint32_t& best, uint32_t& second) {
        uint32_t b = PROJ_NOKEY, s2 = PROJ_NOKEY;
#pragma unroll
        for (int j = 3; j >= 0; j--) {
            const bool open = cr[t[j] & 0xFFFu] >= i;
            s2 = open ? b : s2;
            b = open ? t[j] : b;
        }
        second = best == PROJ_NOKEY ? s2 : b;
        best = best == PROJ_NOKEY ? b : best;
    };
    // whether a key behind 'last' can change what (best, second) decide (with a
    // negative ratio a farther one fails the test where a nearer one passes)
    const bool falling = !(nnratio >= 0.0f);
    auto look_on = [&](uint32_t best, uint32_t second, uint32_t last) {
        return second == PROJ_NOKEY &&
               (best == PROJ_NOKEY ? dist_of(last) <= ORBGPU_TH_HIGH : falling || ratio_fails(best, last));
    };
    auto full_scan = [&](int i, int c, uint32_t& best, uint32_t& second) {
        best = PROJ_NOKEY;
        second = PROJ_NOKEY;
        row_visit(slots + (size_t)i * slot_cap, c, [&](uint32_t key) {
            if (cr[key & 0xFFFu] < i) return;
            const uint32_t hi = max(best, key);
            best = min(best, key);
            second = min(second, hi);
        });
    };
    int rounds = 0;
    bool converged = M == 0;
    for (int round = 0; round <= M + 1 && !converged; round++) {
        rounds = round + 1;
        if (tid == 0) s_flag[(round + 1) % 3] = 0;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < PROJ_MPT; q++) {
            const int i = tid + q * nt;
            if (cnt[q] == 0) continue;  // never assigned
            uint32_t best = PROJ_NOKEY, second = PROJ_NOKEY;
            pick(i, top[q], best, second);
            if (cnt[q] > 4 && look_on(best, second, top[q][3])) {
                const uint4 v = s_next[i];
                const uint32_t t[4] = {v.x, v.y, v.z, v.w};
                pick(i, t, best, second);
                if (cnt[q] > 8 && look_on(best, second, v.w)) full_scan(i, cnt[q], best, second);
            }
            const int r = decide(best, second);
            if (r != res[q]) {
                res[q] = r;
                s_flag[round % 3] = 1;
            }
            if (r >= 0) atomicMin(&cw[r], i);
        }
        for (int i = Mr + tid; i < M; i += nt) {
            uint32_t best, second;
            full_scan(i, min(slot_count[i], slot_cap), best, second);
            const int r = decide(best, second);
            if (r != s_res[i]) {
                s_res[i] = r;
                s_flag[round % 3] = 1;
            }
            if (r >= 0) atomicMin(&cw[r], i);
        }
        __syncthreads();
        converged = s_flag[round % 3] == 0;
        // this round's claims are read by the next; the array read now is cleared for writing
        int* t = cr;
        cr = cw;
        cw = t;
        if (!converged)
            for (int k = tid; k < n; k += nt) cw[k] = cw[k] == -1 ? -1 : PROJ_FREE;
    }
    for (int k = tid; k < n; k += nt) match_out[k] = claimed && claimed[k] ? -2 : -1;
    __syncthreads();
    int nm = 0;
#pragma unroll
    for (int q = 0; q < PROJ_MPT; q++)
        if (cnt[q] > 0 && res[q] >= 0) {
            match_out[res[q]] = tid + q * nt;
            nm++;
        }
    for (int i = Mr + tid; i < M; i += nt) {
        const int r = s_res[i];
        if (r >= 0) {
            match_out[r] = i;
            nm++;
        }
    }
    int tot;
    block_exclusive_scan(nm, s_scan, &tot);
    if (tid == 0) *nmatches = tot;
    return converged ? max(rounds, 1) : 0;
}

}  // namespace orbgpu
