// orbgpu_stereo.cuh -- Frame::ComputeStereoMatches (src/Frame.cc:831-1082) as
// device functions, shared by the per-frame entry (orbgpu_match.cu) and the
// batched one over a batch's resident pyramids (orbgpu_batch.cu).
//
//   row index    one block per pair lists the right keypoints by the row of
//                their y in 16-byte records
//   match        one warp per left keypoint over the records of the rows its
//                octaves' bands [y - 2 scale, y + 2 scale] can reach
//                (src/Frame.cc:875-881; the band itself is tested per record):
//                the best descriptor distance (octave within one level, uR in
//                [uL - maxD, uL]), accepted below (TH_HIGH + TH_LOW) / 2; then
//                the SAD of the centre-subtracted 11 x 11 patch at 11 offsets
//                (22 lanes: each offset's rows in two halves), the first
//                minimum, the parabola, disparity and depth
//                (src/Frame.cc:884-1064)
//   median cut   one block per pair: SADs of the accepted matches at or above
//                1.5 * 1.4 * median discarded (src/Frame.cc:1069-1081)
//
// Bound by latency: a chain of loads per left keypoint.  Listing a keypoint
// once instead of under every row of its band (9 to 30 of them) makes the
// index one launch where counts, scan and fill took three over global memory,
// and a candidate is one record load instead of an index and a 28-byte
// keypoint behind it.
// The patches are read in aligned words (48 loads a lane instead of 132).  The
// median is selected by two histograms of a byte of the SAD (at most 61,710,
// 16 bits); a bitonic sort in global memory took 66 barriers at 2,000 matches.
// A 1241x376 pair with its extractions 452 -> 416 us, 32 pairs 866 -> 843.
// The cut by the last block of the match, one launch less, made every warp of
// the match wait for its stores and its block: the call of 32 pairs 209 us
// against 187 with a launch of its own, of one pair the same.
#pragma once

#include <cuda_fp16.h>

#include "orbgpu_common.cuh"
#include "orbgpu_ext.h"

namespace orbgpu {

struct StereoLevels {
    const uint8_t* left[16];
    const uint8_t* right[16];
    int w[16], h[16], pitch[16];
    float scale[16], inv_scale[16];
    int nlevels;
};

#define STEREO_INDEX_THREADS 1024
#define STEREO_WARPS 8  // left keypoints per block of the match

// The row index of one pair by the calling block (STEREO_INDEX_THREADS
// threads): recs = {x, y, octave, index} of the right keypoints inside the
// pyramid, row by row; start = the rows' first records (nRows + 1 entries,
// nRows at most ORBGPU_MAX_DIM).  A y outside the image counts as its nearest
// row.
__device__ __forceinline__ void stereo_index_block(const orbgpu_keypoint* kpsR, int nR, int nlevels, int nRows,
                                                   int* start, uint4* recs) {
    __shared__ int s_count[ORBGPU_MAX_DIM];
    __shared__ int s_scan[32];
    for (int i = threadIdx.x; i < nRows; i += blockDim.x) s_count[i] = 0;
    __syncthreads();
    const auto row_of = [&](float y) { return min(max((int)floorf(y), 0), nRows - 1); };
    for (int i = threadIdx.x; i < nR; i += blockDim.x)
        if (kpsR[i].octave >= 0 && kpsR[i].octave < nlevels) atomicAdd(&s_count[row_of(kpsR[i].y)], 1);
    __syncthreads();
    int carry = 0;
    for (int b0 = 0; b0 < nRows; b0 += blockDim.x) {
        const int i = b0 + threadIdx.x;
        const int v = i < nRows ? s_count[i] : 0;
        int tot;
        const int ex = block_exclusive_scan(v, s_scan, &tot);
        if (i < nRows) {
            s_count[i] = carry + ex;
            start[i] = carry + ex;
        }
        carry += tot;
    }
    if (threadIdx.x == 0) start[nRows] = carry;
    __syncthreads();
    for (int i = threadIdx.x; i < nR; i += blockDim.x) {
        const float x = kpsR[i].x, y = kpsR[i].y;
        const int oct = kpsR[i].octave;
        if (oct >= 0 && oct < nlevels)
            recs[atomicAdd(&s_count[row_of(y)], 1)] =
                make_uint4(__float_as_uint(x), __float_as_uint(y), (unsigned)oct, (unsigned)i);
    }
}

// 11 bytes of a level's row from column x0 as three words (the last one's top
// byte is not used).  The planes and their pitch are 4-byte aligned, and every
// word read holds a byte of the 11.
__device__ __forceinline__ void stereo_row11(const uint8_t* row, int x0, unsigned (&w)[3]) {
    const unsigned* q = reinterpret_cast<const unsigned*>(row + (x0 & ~3));
    const int o = x0 & 3;
    const unsigned a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    const unsigned d = o >= 2 ? __ldg(q + 3) : 0u;
    w[0] = __funnelshift_r(a, b, 8 * o);
    w[1] = __funnelshift_r(b, c, 8 * o);
    w[2] = __funnelshift_r(c, d, 8 * o);
}

// Bytes 2h and 2h + 1 of a word as 1024 + byte in halves (0x6400 is 1024, its
// last place 1).
template <int H>
__device__ __forceinline__ __half2 stereo_halves(unsigned w) {
    const unsigned v = __byte_perm(w, 0x64646464u, H ? 0x4342 : 0x4140);
    return *reinterpret_cast<const __half2*>(&v);
}

// The match of left keypoint iL, by the calling warp.  Writes uright[iL],
// depth[iL] (-1 when unmatched) and sad_out[iL] (the accepted SAD, -1 none).
__device__ __forceinline__ void stereo_match_warp(int iL, const orbgpu_keypoint* kpsL, const uint8_t* descL,
                                                  const uint8_t* descR, const StereoLevels& lv, int nRows,
                                                  const int* start, const uint4* recs, float bf, float fx,
                                                  float* uright, float* depth, int* sad_out, int* status) {
    const int lane = threadIdx.x & 31;
    float out_ur = -1.0f, out_depth = -1.0f;  // lane 0's
    int out_sad = -1;
    const auto match = [&]() {
        const float uL = kpsL[iL].x, vL = kpsL[iL].y;
        const int levelL = kpsL[iL].octave;
        if (levelL < 0 || levelL >= lv.nlevels) return;
        const int row = (int)vL;
        if (row < 0 || row >= nRows) return;
        // a band of half height r holds the row only if y lies in (row - 1 - r, row + 1 + r)
        float scale = lv.scale[levelL];
        if (levelL > 0) scale = fmaxf(scale, lv.scale[levelL - 1]);
        if (levelL + 1 < lv.nlevels) scale = fmaxf(scale, lv.scale[levelL + 1]);
        const int reach = (int)fminf(fmaxf(ceilf(__fmul_rn(2.0f, scale)), 0.f), (float)nRows);
        const int rs = start[max(row - 1 - reach, 0)], re = start[min(row + reach, nRows - 1) + 1];
        if (rs == re) return;
        const float mb = __fdiv_rn(bf, fx);
        const float minZ = mb, minD = 0.f, maxD = __fdiv_rn(bf, minZ);
        const float minU = __fsub_rn(uL, maxD), maxU = __fsub_rn(uL, minD);
        if (maxU < 0) return;
        // best over the row band: lexicographic (distance, right index), distance < TH_HIGH
        unsigned best = ~0u, best_i = ~0u;
        float best_x = 0.f;
        const uint4* pL = reinterpret_cast<const uint4*>(descL + (size_t)iL * 32);
        const uint4 l0 = __ldg(pL), l1 = __ldg(pL + 1);
        for (int b = rs; b < re; b += 64) {
            uint4 rec[2];
            bool take[2];
            uint4 r0[2], r1[2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int j = b + 32 * u + lane;
                take[u] = j < re;
                if (take[u]) rec[u] = __ldg(recs + j);
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (!take[u]) continue;
                const float x = __uint_as_float(rec[u].x), y = __uint_as_float(rec[u].y);
                const int oct = (int)rec[u].z;
                const float r = __fmul_rn(2.0f, lv.scale[oct]);
                take[u] = oct >= levelL - 1 && oct <= levelL + 1 && x >= minU && x <= maxU &&
                          (int)floorf(__fsub_rn(y, r)) <= row && (int)ceilf(__fadd_rn(y, r)) >= row;
                if (take[u]) {
                    const uint4* pR = reinterpret_cast<const uint4*>(descR + (size_t)rec[u].w * 32);
                    r0[u] = __ldg(pR);
                    r1[u] = __ldg(pR + 1);
                }
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (!take[u]) continue;
                const unsigned dist = hamming256(l0, l1, r0[u], r1[u]);
                if (dist < ORBGPU_TH_HIGH && (dist < best || (dist == best && rec[u].w < best_i))) {
                    best = dist;
                    best_i = rec[u].w;
                    best_x = __uint_as_float(rec[u].x);
                }
            }
        }
        const unsigned bestDist = __reduce_min_sync(0xffffffffu, best);
        const unsigned thOrbDist = (ORBGPU_TH_HIGH + ORBGPU_TH_LOW) / 2;
        if (bestDist >= thOrbDist) return;
        const unsigned bestIdxR = __reduce_min_sync(0xffffffffu, best == bestDist ? best_i : ~0u);
        const unsigned owner = __ballot_sync(0xffffffffu, best == bestDist && best_i == bestIdxR);
        // SAD refinement on the unblurred level (src/Frame.cc:951-1020)
        const float uR0 = __shfl_sync(0xffffffffu, best_x, __ffs(owner) - 1);
        const float sf = lv.inv_scale[levelL];
        const float scaleduL = roundf(__fmul_rn(uL, sf));
        const float scaledvL = roundf(__fmul_rn(vL, sf));
        const float scaleduR0 = roundf(__fmul_rn(uR0, sf));
        constexpr int W = 5, L = 5;
        const int lw = lv.w[levelL], lh = lv.h[levelL], lp = lv.pitch[levelL];
        const float iniu = __fsub_rn(__fsub_rn(scaleduR0, (float)L), (float)W);
        const float endu = __fadd_rn(__fadd_rn(__fadd_rn(scaleduR0, (float)L), (float)W), 1.0f);
        if (iniu < 0 || endu >= (float)lw) return;
        const int ly0 = (int)(scaledvL - W), lx0 = (int)(scaleduL - W);
        if (ly0 < 0 || ly0 + 2 * W + 1 > lh || lx0 < 0 || lx0 + 2 * W + 1 > lw) {
            if (lane == 0) atomicOr(status, 1);
            return;
        }
        const uint8_t* left = lv.left[levelL] + (size_t)ly0 * lp;
        const uint8_t* right = lv.right[levelL] + (size_t)ly0 * lp;
        // offset t = incR + L on lanes t and t + 11: rows 0-5 and rows 6-10
        // In halves: l - r - c is at most 510, four of them sum to at most 2,040,
        // and integers up to 2,048 are exact.  In integers a pixel took 5
        // instructions of the ALU pipe: the call of 32 pairs 187 us against 169.
        float part = 0.f;
        if (lane < 2 * (2 * L + 1)) {
            const bool upper = lane < 2 * L + 1;
            const int t = upper ? lane : lane - (2 * L + 1);
            const int rx0 = (int)(scaleduR0 + (t - L) - W);
            const int c = (int)left[(size_t)W * lp + lx0 + W] - (int)right[(size_t)W * lp + rx0 + W];
            const __half2 c2 = __half2half2(__int2half_rn(c));
            const uint8_t* lr = left + (upper ? 0 : (size_t)(W + 1) * lp);
            const uint8_t* rr = right + (upper ? 0 : (size_t)(W + 1) * lp);
#pragma unroll
            for (int yy = 0; yy < W + 1; yy++) {
                if (yy == W && !upper) break;
                unsigned a[3], b[3];
                stereo_row11(lr + (size_t)yy * lp, lx0, a);
                stereo_row11(rr + (size_t)yy * lp, rx0, b);
                const auto diff = [&](__half2 l, __half2 r) { return __habs2(__hsub2(__hsub2(l, r), c2)); };
                const __half2 s8 = __hadd2(__hadd2(diff(stereo_halves<0>(a[0]), stereo_halves<0>(b[0])),
                                                   diff(stereo_halves<1>(a[0]), stereo_halves<1>(b[0]))),
                                           __hadd2(diff(stereo_halves<0>(a[1]), stereo_halves<0>(b[1])),
                                                   diff(stereo_halves<1>(a[1]), stereo_halves<1>(b[1]))));
                const __half2 s2 = diff(stereo_halves<0>(a[2]), stereo_halves<0>(b[2]));
                const __half2 s1 = diff(stereo_halves<1>(a[2]), stereo_halves<1>(b[2]));  // column 10, and one past it
                const float2 f8 = __half22float2(s8), f3 = __half22float2(__hadd2(s2, __halves2half2(__low2half(s1), __ushort_as_half(0))));
                part += f8.x + f8.y + f3.x + f3.y;
            }
        }
        const float other = __shfl_down_sync(0xffffffffu, part, 2 * L + 1);
        // first minimum over incR = -L..L: SAD (16 bits), then the offset
        const unsigned key = lane < 2 * L + 1 ? (unsigned)(int)(part + other) << 4 | (unsigned)lane : ~0u;
        const unsigned least = __reduce_min_sync(0xffffffffu, key);
        const int t = (int)(least & 15), bestinc = t - L;
        if (bestinc == -L || bestinc == L) return;
        const float d1 = (float)(__shfl_sync(0xffffffffu, key, t - 1) >> 4), d2 = (float)(least >> 4),
                    d3 = (float)(__shfl_sync(0xffffffffu, key, t + 1) >> 4);
        const float deltaR = __fdiv_rn(__fsub_rn(d1, d3), __fmul_rn(2.0f, __fsub_rn(__fadd_rn(d1, d3), __fmul_rn(2.0f, d2))));
        if (deltaR < -1 || deltaR > 1) return;
        float bestuR = __fmul_rn(lv.scale[levelL], __fadd_rn(__fadd_rn(scaleduR0, (float)bestinc), deltaR));
        float disparity = __fsub_rn(uL, bestuR);
        if (disparity >= minD && disparity < maxD) {
            if (disparity <= 0) {
                disparity = 0.01f;
                bestuR = (float)((double)uL - 0.01);
            }
            out_depth = __fdiv_rn(bf, disparity);
            out_ur = bestuR;
            out_sad = (int)(least >> 4);
        }
    };
    match();
    if (lane == 0) {
        uright[iL] = out_ur;
        depth[iL] = out_depth;
        sad_out[iL] = out_sad;
    }
}

// Element k of the counts in hist[256] (the first bin at which the running
// count passes k) by the calling warp; k becomes the rank inside the bin.
__device__ __forceinline__ int stereo_select_bin(const int* hist, int& k) {
    const int lane = threadIdx.x & 31;
    int own[8], sum = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        own[i] = hist[8 * lane + i];
        sum += own[i];
    }
    int incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    const int src = __ffs(__ballot_sync(0xffffffffu, incl > k)) - 1;
    int bin = 8 * lane, rest = k - (incl - sum);
#pragma unroll
    for (int i = 0; i < 7; i++)
        if (bin == 8 * lane + i && rest >= own[i]) {
            rest -= own[i];
            bin++;
        }
    k = __shfl_sync(0xffffffffu, rest, src);
    return __shfl_sync(0xffffffffu, bin, src);
}

// The median cut of one pair's nL left keypoints by the calling block.
__device__ __forceinline__ void stereo_median_block(int nL, const int* sad, float* uright, float* depth) {
    __shared__ int s_hist[2][256];
    __shared__ int s_at[2];
    __shared__ int s_cnt;
    for (int i = threadIdx.x; i < 512; i += blockDim.x) s_hist[i >> 8][i & 255] = 0;
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    int cnt = 0;
    for (int i = threadIdx.x; i < nL; i += blockDim.x) {
        const int v = sad[i];
        if (v >= 0) {
            cnt++;
            atomicAdd(&s_hist[0][v >> 8], 1);
        }
    }
    atomicAdd(&s_cnt, cnt);
    __syncthreads();
    if (s_cnt == 0) return;
    int k = s_cnt / 2;
    if (threadIdx.x < 32) {
        const int bin = stereo_select_bin(s_hist[0], k);
        if (threadIdx.x == 0) s_at[0] = bin;
    }
    __syncthreads();
    const int high = s_at[0];
    for (int i = threadIdx.x; i < nL; i += blockDim.x) {
        const int v = sad[i];
        if (v >= 0 && (v >> 8) == high) atomicAdd(&s_hist[1][v & 255], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int bin = stereo_select_bin(s_hist[1], k);
        if (threadIdx.x == 0) s_at[1] = bin;
    }
    __syncthreads();
    const float median = (float)(high << 8 | s_at[1]);
    const float thDist = __fmul_rn(1.5f * 1.4f, median);
    for (int i = threadIdx.x; i < nL; i += blockDim.x) {
        const int v = sad[i];
        if (v >= 0 && !((float)v < thDist)) {
            uright[i] = -1.0f;
            depth[i] = -1.0f;
        }
    }
}

}  // namespace orbgpu
