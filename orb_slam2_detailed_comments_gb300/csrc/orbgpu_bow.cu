// orbgpu_bow.cu -- DBoW2's vocabulary transform (Frame::ComputeBoW,
// src/Frame.cc:704-718: ORBVocabulary::transform(descriptors, mBowVec,
// mFeatVec, 4)) for the features of many frames.
//
// The vocabulary tree lives in HBM with every node's children contiguous
// (grouped by parent in node-id order, the order loadFromTextFile appends
// them), so one descent level reads the k child descriptors of one node as
// consecutive 32-byte rows.  k_bow_descend: 8 lanes per feature walk the
// tree (TemplatedVocabulary.h:1240-1290: at every level the first child with
// the least Hamming distance, strict <; the node of level L - levelsup kept
// for the feature vector; stop at a node without children) and write the
// word, its weight and that node.  k_bow_assemble: two blocks per frame sort
// the kept features (weight > 0) by word and by node in shared memory and
// writes BowVector (BowVector::addWeight / addIfNotExist, then normalize,
// BowVector.cpp:40-95) and FeatureVector (FeatureVector::addFeature,
// FeatureVector.cpp:37-53).  The doubles are the reference's: a word seen c
// times sums its weight c times in sequence (the reference adds them in
// feature order, and they are equal), and the norm is one sequential sum in
// ascending word order, as std::map iterates.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <sstream>
#include <string>
#include <vector>

#include "orbgpu_host.h"

struct orbgpu_vocabulary {
    int k, L, scoring, weighting, nnodes, nwords;
    uint4* child_desc;   // one 32-byte row per non-root node, grouped by parent
    int4* child_info;    // per position: node id, its children's positions [y, z), word id (0 where none, as DBoW2's Node)
    double* node_weight;
    int root_end;        // the root's children are positions [0, root_end)
};

namespace orbgpu {

#define BOW_THREADS 256
#define BOW_ASM_THREADS 1024
#define BOW_MAX_FEATURES 8192  // per frame (the assembly sorts a frame in shared memory)

// Bound by the latency of the levels (two dependent loads each) and by POPC.
// A lane takes half a child's row, so the 8 lanes of a feature read 4
// children's 128 bytes at once; a thread per feature touched 32 lines with
// every load, and asked three arrays for a node where child_info is one load
// (128,000 features in ten children and six levels: 48 -> 40 us).
__global__ void __launch_bounds__(BOW_THREADS) k_bow_descend(const uint4* __restrict__ desc, const int* __restrict__ offsets,
                                                             int nframes, const uint4* __restrict__ child_desc,
                                                             const int4* __restrict__ child_info, int root_end,
                                                             const double* __restrict__ node_weight, int nid_level,
                                                             int* __restrict__ word_out, double* __restrict__ weight_out,
                                                             int* __restrict__ node_out) {
    const int first = __ldg(offsets), last = __ldg(offsets + nframes);
    if (first < 0) return;
    const int l = threadIdx.x & 7;
    const unsigned group = 0xffu << (threadIdx.x & 24);
    for (int i = first + (blockIdx.x * BOW_THREADS + threadIdx.x) / 8; i < last; i += gridDim.x * (BOW_THREADS / 8)) {
        const uint4 f = __ldg(desc + 2 * (size_t)i + (l & 1));
        int4 at = make_int4(0, 0, root_end, 0);  // the root
        int level = 0, nid = 0;
        while (at.y < at.z) {
            ++level;
            int best_d = 512, best = 0;
            for (int c0 = at.y; c0 < at.z; c0 += 4) {
                const int c = c0 + (l >> 1);
                int d = 0;
                if (c < at.z) {
                    const uint4 r = __ldg(child_desc + 2 * (size_t)c + (l & 1));
                    d = __popc(f.x ^ r.x) + __popc(f.y ^ r.y) + __popc(f.z ^ r.z) + __popc(f.w ^ r.w);
                }
                d += __shfl_xor_sync(group, d, 1);
                if (c < at.z && d < best_d) {
                    best_d = d;
                    best = c;
                }
            }
#pragma unroll
            for (int o = 2; o <= 4; o <<= 1) {
                const int d = __shfl_xor_sync(group, best_d, o), c = __shfl_xor_sync(group, best, o);
                if (d < best_d || (d == best_d && c < best)) {
                    best_d = d;
                    best = c;
                }
            }
            at = __ldg(child_info + best);
            if (level == nid_level) nid = at.x;
        }
        if (l == 0) {
            word_out[i] = at.w;
            weight_out[i] = __ldg(node_weight + at.x);
            node_out[i] = nid;
        }
    }
}

// Ascending bitonic sort of n2 (a power of two, at least 32) 64-bit keys in
// shared memory.  Strides below 32 stay in a warp's registers: 21 of the 66
// steps of 2,048 keys go through shared memory and a barrier.
__device__ void bow_block_sort(unsigned long long* keys, int n2) {
    const int lane = threadIdx.x & 31;
    // the strides from 'from' (at most 16) down of the merges of sizes k0 .. k1
    const auto in_warp = [&](int k0, int k1, int from) {
        for (int b = threadIdx.x - lane; b < n2; b += blockDim.x) {
            const int i = b + lane;
            unsigned long long key = keys[i];
            for (int k = k0; k <= k1; k <<= 1)
                for (int j = min(k >> 1, from); j > 0; j >>= 1) {
                    const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, j);
                    const bool low = ((i & j) == 0) == ((i & k) == 0);
                    key = (other < key) == low ? other : key;
                }
            keys[i] = key;
        }
        __syncthreads();
    };
    in_warp(2, 32, 16);
    for (int k = 64; k <= n2; k <<= 1) {
        for (int j = k >> 1; j >= 32; j >>= 1) {
            for (int t = threadIdx.x; t < n2 / 2; t += blockDim.x) {
                const int i = 2 * t - (t & (j - 1)), l = i + j;
                const unsigned long long a = keys[i], b = keys[l];
                if ((a > b) == ((i & k) == 0)) {
                    keys[i] = b;
                    keys[l] = a;
                }
            }
            __syncthreads();
        }
        in_warp(k, k, 16);
    }
}

// The sum of n terms (not negative) in ascending order, each addition rounded,
// as a loop over doubles gives it, by one warp.  While the sum s stays within
// one power of two, adding x adds x rounded to s's unit in the last place: an
// integer that does not depend on s except where x lies halfway.  So 32 terms
// become integers and are summed at once (by a scan where one of them is not
// such a term); only a term that is halfway, is larger than s's power of two,
// carries s past it or is not a normal number is added as a double (about two
// per power of two of the sum).  The loop over doubles waits some 50 cycles a term for the FP64 pipe: 64 frames of 2,000
// features took 104 us to assemble and take 46.
template <bool SQUARES>
__device__ double bow_sequential_sum(const double* v, int n) {
    const int lane = threadIdx.x & 31;
    const unsigned long long one = 1ull << 52, frac = one - 1;
    const auto load = [&](int i) {
        if (i >= n) return 0.0;
        const double x = v[i];
        return SQUARES ? __dmul_rn(x, x) : fabs(x);
    };
    double s = 0.0, next = load(lane);
    for (int base = 0; base < n; base += 32) {
        const double x = next;
        next = load(base + 32 + lane);
        const unsigned long long xb = __double_as_longlong(x);
        const int ex = (int)(xb >> 52) & 0x7ff;
        const unsigned long long mx = (xb & frac) | one;
        unsigned todo = __ballot_sync(0xffffffffu, x != 0.0);  // a zero changes nothing
        while (todo) {
            const unsigned long long sb = __double_as_longlong(s);
            const int es = (int)(sb >> 52) & 0x7ff;
            const unsigned long long ms = (sb & frac) | one;
            const bool mine = (todo >> lane) & 1u;
            const int d = es - ex;
            bool alone = ex == 0 || ex == 0x7ff || es == 0 || es == 0x7ff || d < 0;
            unsigned long long q = 0;
            if (mine && !alone && d <= 53) {
                const unsigned long long rest = mx & ((1ull << d) - 1), half = (1ull << d) >> 1;
                q = (mx >> d) + (rest > half ? 1 : 0);
                alone = d > 0 && rest == half;
            }
            // the usual case: all 32 (of 54 bits, summed in two halves) at once
            const unsigned any_alone = __ballot_sync(0xffffffffu, mine && alone);
            const unsigned long long sum =
                ((unsigned long long)__reduce_add_sync(0xffffffffu, (unsigned)(q >> 27)) << 27) +
                __reduce_add_sync(0xffffffffu, (unsigned)q & ((1u << 27) - 1u));
            if (!any_alone && ms + sum < 2 * one) {
                if (sum) s = __longlong_as_double((long long)(((unsigned long long)es << 52) | ((ms + sum) & frac)));
                break;
            }
            unsigned long long incl = q;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            // the first term that is added as a double, and the integers before it
            const unsigned event = __ballot_sync(0xffffffffu, mine && (alone || ms + incl >= 2 * one));
            const int f = __ffs(event) - 1;
            const unsigned long long add = __shfl_sync(0xffffffffu, incl - q, f);
            if (add) s = __longlong_as_double((long long)(((unsigned long long)es << 52) | ((ms + add) & frac)));
            s = __dadd_rn(s, __shfl_sync(0xffffffffu, x, f));
            todo &= ~((2u << f) - 1u);
        }
    }
    return s;
}

// Two blocks per frame (block 2f builds frame f's BowVector, block 2f + 1 its
// FeatureVector).  Shared memory: BOW_MAX_FEATURES 64-bit keys per block.
__global__ void __launch_bounds__(BOW_ASM_THREADS) k_bow_assemble(
    const int* __restrict__ offsets, const int* __restrict__ word, const double* __restrict__ weight,
    const int* __restrict__ node, int weighting, int scoring, int* __restrict__ bow_counts,
    int* __restrict__ bow_words, double* __restrict__ bow_values, int* __restrict__ fv_counts,
    int* __restrict__ fv_nodes, int* __restrict__ fv_starts, int* __restrict__ fv_sizes,
    int* __restrict__ fv_features) {
    extern __shared__ unsigned long long keys[];
    __shared__ int s_nkept;
    __shared__ double s_norm;
    // two blocks per frame: pass 0 the BowVector (keys word << 32 | feature),
    // pass 1 the FeatureVector (node << 32 | feature)
    const int f = blockIdx.x >> 1, pass = blockIdx.x & 1;
    const int o0 = offsets[f], o1 = offsets[f + 1];
    const int n = o1 - o0;
    if (o0 < 0 || n < 0 || n > BOW_MAX_FEATURES) {
        if (threadIdx.x == 0) (pass == 0 ? bow_counts : fv_counts)[f] = -1;
        return;
    }
    int n2 = 32;
    while (n2 < n) n2 <<= 1;
    const unsigned long long pad = ~0ull;
    {
        for (int i = threadIdx.x; i < n2; i += blockDim.x) {
            unsigned long long key = pad;
            if (i < n && weight[o0 + i] > 0.0) {
                const unsigned hi = pass == 0 ? (unsigned)word[o0 + i] : (unsigned)node[o0 + i];
                key = ((unsigned long long)hi << 32) | (unsigned)i;
            }
            keys[i] = key;
        }
        if (threadIdx.x == 0) s_nkept = 0;
        __syncthreads();
        bow_block_sort(keys, n2);
        // kept features sort first; runs of equal high words are the entries
        int kept = 0;
        for (int i = threadIdx.x; i < n2; i += blockDim.x) kept += keys[i] != pad ? 1 : 0;
        kept = __reduce_add_sync(0xffffffffu, kept);
        if ((threadIdx.x & 31) == 0 && kept) atomicAdd(&s_nkept, kept);
        __syncthreads();
        const int nk = s_nkept;
        // run starts in ascending order: a block-wide exclusive scan of the flags
        __shared__ int s_scan[BOW_ASM_THREADS / 32];
        int nruns = 0;
        for (int base = 0; base < nk; base += blockDim.x) {
            const int i = base + threadIdx.x;
            const bool start = i < nk && (i == 0 || (keys[i] >> 32) != (keys[i - 1] >> 32));
            int tot;
            const int r = nruns + block_exclusive_scan(start ? 1 : 0, s_scan, &tot);
            nruns += tot;
            if (start) {
                int end = i + 1;
                while (end < nk && (keys[end] >> 32) == (keys[i] >> 32)) end++;
                const unsigned hi = (unsigned)(keys[i] >> 32);
                if (pass == 0) {
                    const double w0 = weight[o0 + (int)(keys[i] & 0xffffffffu)];
                    double v = w0;
                    if (weighting == 0 || weighting == 1)  // TF_IDF, TF: addWeight per occurrence
                        for (int q = i + 1; q < end; q++) v = __dadd_rn(v, w0);
                    bow_words[o0 + r] = (int)hi;
                    bow_values[o0 + r] = v;
                } else {
                    fv_nodes[o0 + r] = (int)hi;
                    fv_starts[o0 + r] = o0 + i;
                    fv_sizes[o0 + r] = end - i;
                }
            }
        }
        if (pass == 1) {
            // the features of every node, in feature order (the sort's low words)
            for (int i = threadIdx.x; i < nk; i += blockDim.x) fv_features[o0 + i] = (int)(keys[i] & 0xffffffffull);
            if (threadIdx.x == 0) fv_counts[f] = nruns;
            return;
        }
        // normalisation (ScoringObject.h:84-89: L1 for L1 / chi-square / KL /
        // Bhattacharyya, L2 for L2, none for the dot product, where TF divides
        // by the number of words instead)
        __syncthreads();
        if (threadIdx.x < 32) {
            double norm = 0.0;
            if (scoring == 5) {
                norm = (weighting == 0 || weighting == 1) && nruns > 0 ? (double)nruns : 0.0;
            } else if (scoring == 1) {
                norm = __dsqrt_rn(bow_sequential_sum<true>(bow_values + o0, nruns));
            } else {
                norm = bow_sequential_sum<false>(bow_values + o0, nruns);
            }
            if (threadIdx.x == 0) {
                s_norm = norm;
                bow_counts[f] = nruns;
            }
        }
        __syncthreads();
        const double norm = s_norm;
        if (norm > 0.0)
            for (int r = threadIdx.x; r < nruns; r += blockDim.x) bow_values[o0 + r] = __ddiv_rn(bow_values[o0 + r], norm);
        __syncthreads();
    }
}

// ORBmatcher::SearchByBoW(KeyFrame* pKF, Frame& F, vpMapPointMatches),
// src/ORBmatcher.cc:247-380, one cluster of 8 blocks per (keyframe, frame)
// pair.  A frame feature belongs to one FeatureVector node and so does a
// keyframe feature: the nodes both vectors hold are independent, and one warp
// takes one node (found by a 32-way search in the keyframe's sorted node list).
// Inside a node the keyframe features run in list order, as in the reference:
// each takes, among the node's frame features not matched yet, the first at
// the least distance, with the second-best over the rest; kept when
// best <= TH_LOW and best < nnratio * second.  Then the rotation histogram
// (block 0's shared memory), ComputeThreeMaxima (src/ORBmatcher.cc:2035-2077)
// and the resets.  MODE 1 is SearchByBoW(KeyFrame* pKF1, KeyFrame* pKF2,
// vpMatches12) (src/ORBmatcher.cc:729-880): candidates need a map point that
// is not bad, TH_LOW is exclusive, and the result is per pKF1 feature.
// MODE 2: SearchForTriangulation.
//
// Bound by latency: a node's features are taken one after the other.  A lane
// holds two frame features' descriptors (nodes of more than 64 read theirs
// again for every keyframe feature) and one keyframe feature's, passed round
// by shuffles, so a turn waits for no memory; a pair's nodes are spread over 8
// SMs.  32 pairs of 2,000 features: 98 us with a block per pair that read both
// features from memory every turn, 48 with one frame feature a lane (nodes of
// more than 32 then set the time), 38 with two.
#define SBB_THREADS 256
#define SBB_CLUSTER 8
#define SBB_HELD 64  // frame features of a node in a warp's registers
#define SBB_TH_LOW 50

// SearchForTriangulation's per-call constants: pKF2's scale tables (read at
// the candidate's octave) and bOnlyStereo.
struct TriangulationDev {
    float scale[16];
    float sigma2[16];
    int only_stereo;
};

template <int MODE>
__global__ void __launch_bounds__(SBB_THREADS) k_search_by_bow(
    const orbgpu_keypoint* __restrict__ kps, const uint4* __restrict__ desc, const int* __restrict__ offsets,
    const int* __restrict__ fv_counts, const int* __restrict__ fv_nodes, const int* __restrict__ fv_starts,
    const int* __restrict__ fv_sizes, const int* __restrict__ fv_features, const uint8_t* __restrict__ kf_mp,
    const int* __restrict__ pairs, float nnratio, int check_ori, const float* __restrict__ pair_params,
    const float* __restrict__ uright, const __grid_constant__ TriangulationDev tri, const int* __restrict__ out_offsets,
    int* match_out, int* __restrict__ nmatches) {
    constexpr bool TRIANG = MODE == 2;
    __shared__ unsigned s_taken[BOW_MAX_FEATURES / 32];  // of nodes with more than SBB_HELD frame features
    __shared__ unsigned char s_bin[BOW_MAX_FEATURES];    // block 0's: every match's bin
    __shared__ int s_hist[32];                           // block 0's
    __shared__ int s_total[32];
    __shared__ int s_ind[3], s_nm;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int p = blockIdx.x / SBB_CLUSTER;
    const int kf = pairs[2 * p], fr = pairs[2 * p + 1];
    const int ok0 = offsets[kf], of0 = offsets[fr];
    const int kn = offsets[kf + 1] - ok0, frn = offsets[fr + 1] - of0;
    // the output (and bins) are per frame feature, or per first-keyframe
    // feature for two keyframes (vpMatches12)
    const int fn = MODE ? kn : frn;
    const int ckf = fv_counts[kf], cf = fv_counts[fr];
    int* out = match_out + out_offsets[p];
    if (kn < 0 || kn > BOW_MAX_FEATURES || frn < 0 || frn > BOW_MAX_FEATURES || ckf < 0 || cf < 0) {
        if (rank == 0 && threadIdx.x == 0) nmatches[p] = -1;
        return;
    }
    const int first = rank * SBB_THREADS + threadIdx.x;
    for (int i = first; i < fn; i += SBB_CLUSTER * SBB_THREADS) out[i] = -1;
    for (int i = threadIdx.x; i < BOW_MAX_FEATURES / 32; i += SBB_THREADS) s_taken[i] = 0;
    if (threadIdx.x < 32) s_hist[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_nm = 0;
    unsigned char* bins = cluster.map_shared_rank(s_bin, 0);
    int* hist = cluster.map_shared_rank(s_hist, 0);
    cluster.sync();
    const int lane = threadIdx.x & 31;
    // F12 (row-major) and the epipole in pKF2
    float F[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, ex = 0.f, ey = 0.f;
    if (TRIANG) {
#pragma unroll
        for (int q = 0; q < 9; q++) F[q] = pair_params[11 * p + q];
        ex = pair_params[11 * p + 9];
        ey = pair_params[11 * p + 10];
    }
    const float factor = __fdiv_rn((float)ORBGPU_HISTO_LENGTH, 360.0f);
    const unsigned INF = 0x7fffffffu;
    // neighbouring nodes, which are of like size, go to different SMs
    for (int j = (threadIdx.x >> 5) * SBB_CLUSTER + rank; j < cf; j += SBB_CLUSTER * SBB_THREADS / 32) {
        const int node = fv_nodes[of0 + j];
        int lo = 0, len = ckf, jk = -1;
        while (len > 0) {
            const int step = (len + 31) >> 5, at = lane * step;
            const int v = at < len ? fv_nodes[ok0 + lo + at] : 0x7fffffff;
            const unsigned same = __ballot_sync(0xffffffffu, at < len && v == node);
            const int below = __popc(__ballot_sync(0xffffffffu, at < len && v < node));
            if (same) {
                jk = lo + (__ffs(same) - 1) * step;
                break;
            }
            if (below == 0) break;
            const int skip = (below - 1) * step + 1;
            lo += skip;
            len = min(step - 1, len - skip);
        }
        if (jk < 0) continue;
        const int* flist = fv_features + fv_starts[of0 + j];
        const int fcount = fv_sizes[of0 + j];
        const int* klist = fv_features + fv_starts[ok0 + jk];
        const int kcount = fv_sizes[ok0 + jk];
        // the lane's frame features c + lane and c + 32 + lane
        int jf[2] = {0, 0};
        uint4 f0[2], f1[2];
        bool open[2], st2[2] = {false, false};
        float x2[2], y2[2], angle2[2] = {0.f, 0.f};
        int octave2[2];
        const auto load = [&](int c) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                open[u] = false;
                if (c + 32 * u + lane >= fcount) continue;
                const int i = flist[c + 32 * u + lane];
                jf[u] = i;
                if (MODE == 1 && kf_mp[of0 + i] != 1) continue;
                if (TRIANG) {
                    st2[u] = uright[of0 + i] >= 0.0f;
                    if (kf_mp[of0 + i] != 0 || (tri.only_stereo && !st2[u])) continue;
                    x2[u] = kps[of0 + i].x;
                    y2[u] = kps[of0 + i].y;
                    octave2[u] = kps[of0 + i].octave;
                }
                open[u] = fcount <= SBB_HELD || !((s_taken[i >> 5] >> (i & 31)) & 1u);
                f0[u] = __ldg(desc + 2 * (size_t)(of0 + i));
                f1[u] = __ldg(desc + 2 * (size_t)(of0 + i) + 1);
                if (check_ori) angle2[u] = kps[of0 + i].angle;
            }
        };
        if (fcount <= SBB_HELD) load(0);
        for (int t0 = 0; t0 < kcount; t0 += 32) {
            // the lane's keyframe feature
            int ik = 0;
            uint4 k0 = make_uint4(0, 0, 0, 0), k1 = k0;
            bool use = false, stereo1 = false;
            float angle1 = 0.f, px = 0.f, py = 0.f;
            if (t0 + lane < kcount) {
                ik = klist[t0 + lane];
                use = kf_mp[ok0 + ik] == (TRIANG ? 0 : 1);
                if (TRIANG) {
                    // features without a map point (bad or not), stereo ones only with bOnlyStereo
                    stereo1 = uright[ok0 + ik] >= 0.0f;
                    use = use && (!tri.only_stereo || stereo1);
                    px = kps[ok0 + ik].x;
                    py = kps[ok0 + ik].y;
                }
                if (use) {
                    k0 = __ldg(desc + 2 * (size_t)(ok0 + ik));
                    k1 = __ldg(desc + 2 * (size_t)(ok0 + ik) + 1);
                    if (check_ori) angle1 = kps[ok0 + ik].angle;
                }
            }
            unsigned todo = __ballot_sync(0xffffffffu, use);
            while (todo) {
                const int t = __ffs(todo) - 1;
                todo &= todo - 1;
                const auto from = [&](unsigned v) { return __shfl_sync(0xffffffffu, v, t); };
                const uint4 a0 = make_uint4(from(k0.x), from(k0.y), from(k0.z), from(k0.w));
                const uint4 a1 = make_uint4(from(k1.x), from(k1.y), from(k1.z), from(k1.w));
                bool st1 = false;
                float la = 0.f, lb = 0.f, lc = 0.f;
                if (TRIANG) {
                    st1 = __shfl_sync(0xffffffffu, (int)stereo1, t) != 0;
                    const float x1 = __shfl_sync(0xffffffffu, px, t), y1 = __shfl_sync(0xffffffffu, py, t);
                    // CheckDistEpipolarLine (src/ORBmatcher.cc:205-232): the line of kp1 in pKF2
                    la = __fadd_rn(__fadd_rn(__fmul_rn(x1, F[0]), __fmul_rn(y1, F[3])), F[6]);
                    lb = __fadd_rn(__fadd_rn(__fmul_rn(x1, F[1]), __fmul_rn(y1, F[4])), F[7]);
                    lc = __fadd_rn(__fadd_rn(__fmul_rn(x1, F[2]), __fmul_rn(y1, F[5])), F[8]);
                }
                unsigned b1 = INF;
                int b2 = 256;
                for (int c = 0; c < fcount; c += SBB_HELD) {
                    if (fcount > SBB_HELD) load(c);
                    unsigned key[2] = {INF, INF};
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        if (!open[u]) continue;
                        const int dd = hamming256(a0, a1, f0[u], f1[u]);
                        bool ok = true;
                        if (TRIANG) {
                            ok = dd <= SBB_TH_LOW && octave2[u] >= 0 && octave2[u] < 16;
                            if (ok && !st1 && !st2[u]) {
                                const float dx = __fsub_rn(ex, x2[u]), dy = __fsub_rn(ey, y2[u]);
                                if (__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)) <
                                    __fmul_rn(100.0f, tri.scale[octave2[u]]))
                                    ok = false;
                            }
                            if (ok) {
                                const float num = __fadd_rn(__fadd_rn(__fmul_rn(la, x2[u]), __fmul_rn(lb, y2[u])), lc);
                                const float den = __fadd_rn(__fmul_rn(la, la), __fmul_rn(lb, lb));
                                ok = den != 0.0f && (double)__fdiv_rn(__fmul_rn(num, num), den) <
                                                        __dmul_rn(3.84, (double)tri.sigma2[octave2[u]]);
                            }
                        }
                        // triangulation: the last candidate at the least distance wins ("dist > bestDist" skips)
                        const int i = c + 32 * u + lane;
                        if (ok) key[u] = ((unsigned)dd << 13) | (unsigned)(TRIANG ? 8191 - i : i);
                    }
                    const unsigned c1 = __reduce_min_sync(0xffffffffu, min(key[0], key[1]));
                    // a lone group beyond TH_LOW is not taken whatever its second
                    if (TRIANG || (fcount <= SBB_HELD && c1 >> 13 > SBB_TH_LOW)) {
                        b1 = min(b1, c1);
                        continue;
                    }
                    const unsigned other = key[0] == c1 ? key[1] : key[1] == c1 ? key[0] : min(key[0], key[1]);
                    const int c2 = (int)min(__reduce_min_sync(0xffffffffu, other) >> 13, 256u);
                    if (c1 < b1) {
                        b2 = min(b1 == INF ? 256 : (int)(b1 >> 13), c2);
                        b1 = c1;
                    } else {
                        b2 = min(b2, c1 == INF ? 256 : (int)(c1 >> 13));
                    }
                }
                const int best1 = b1 == INF ? 256 : (int)(b1 >> 13);
                // TH_LOW inclusive for (keyframe, frame), exclusive for two
                // keyframes; triangulation: any candidate left (no ratio test)
                const bool take = TRIANG ? b1 != INF
                                         : (MODE ? best1 < SBB_TH_LOW : best1 <= SBB_TH_LOW) &&
                                               (float)best1 < __fmul_rn(nnratio, (float)b2);
                if (!take) continue;
                const int at = (int)(TRIANG ? 8191u - (b1 & 8191u) : b1 & 8191u);
                const int ikf = __shfl_sync(0xffffffffu, ik, t);
                const float a = __shfl_sync(0xffffffffu, angle1, t);
                if (fcount > SBB_HELD) load(at & ~(SBB_HELD - 1));
                if (lane == (at & 31)) {
                    const bool second = (at & 32) != 0;
                    const int i = second ? jf[1] : jf[0];
                    if (second) open[1] = false;
                    else open[0] = false;
                    if (fcount > SBB_HELD) atomicOr(&s_taken[i >> 5], 1u << (i & 31));
                    const int slot = MODE ? ikf : i;
                    out[slot] = MODE ? i : ikf;  // modes 1 and 2 report per first-keyframe feature
                    if (check_ori) {
                        float rot = __fsub_rn(a, second ? angle2[1] : angle2[0]);
                        if (rot < 0.0f) rot = __fadd_rn(rot, 360.0f);
                        int bin = (int)roundf(__fmul_rn(rot, factor));
                        if (bin == ORBGPU_HISTO_LENGTH) bin = 0;
                        bins[slot] = (unsigned char)bin;
                        atomicAdd(&hist[bin], 1);
                    }
                }
                __syncwarp();
            }
        }
    }
    cluster.sync();
    if (threadIdx.x < 32) s_total[threadIdx.x] = hist[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) {
        int ind1 = -1, ind2 = -1, ind3 = -1;
        if (check_ori) {
            int max1 = 0, max2 = 0, max3 = 0;
            for (int b = 0; b < ORBGPU_HISTO_LENGTH; b++) {  // ComputeThreeMaxima, src/ORBmatcher.cc:2035-2077
                const int sz = s_total[b];
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
    int kept = 0;
    for (int i = first; i < fn; i += SBB_CLUSTER * SBB_THREADS) {
        if (__ldcg(out + i) < 0) continue;
        if (check_ori) {
            const int b = bins[i];
            if (b != s_ind[0] && b != s_ind[1] && b != s_ind[2]) {
                out[i] = -1;
                continue;
            }
        }
        kept++;
    }
    kept = __reduce_add_sync(0xffffffffu, kept);
    if (lane == 0 && kept) atomicAdd(cluster.map_shared_rank(&s_nm, 0), kept);
    cluster.sync();
    if (rank == 0 && threadIdx.x == 0) nmatches[p] = s_nm;
}

}  // namespace orbgpu

using namespace orbgpu;

static int search_by_bow(const orbgpu_keypoint* kps, const uint8_t* desc, const int* offsets, const int* fv_counts,
                         const int* fv_nodes, const int* fv_starts, const int* fv_sizes, const int* fv_features,
                         const uint8_t* kf_mappoints, const int* pairs, int npairs, float nnratio, int check_ori,
                         int keyframes, const int* out_offsets, int* match_out, int* nmatches, void* stream,
                         const float* pair_params = nullptr, const float* uright = nullptr,
                         const TriangulationDev* tri = nullptr) {
    if (npairs < 0 || (npairs > 0 && (!kps || !desc || !offsets || !fv_counts || !fv_nodes || !fv_starts ||
                                      !fv_sizes || !fv_features || !kf_mappoints || !pairs || !out_offsets ||
                                      !match_out || !nmatches)) ||
        ((uintptr_t)desc & 15)) {
        orbgpu_set_last_error("orbgpu_search_by_bow: bad arguments", __FILE__, __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    if (npairs == 0) return ORBGPU_OK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)npairs * SBB_CLUSTER);
    cfg.blockDim = dim3(SBB_THREADS);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = SBB_CLUSTER;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const auto kernel = keyframes == 0 ? k_search_by_bow<0> : keyframes == 1 ? k_search_by_bow<1> : k_search_by_bow<2>;
    ORBGPU_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, kps, reinterpret_cast<const uint4*>(desc), offsets, fv_counts, fv_nodes,
                                       fv_starts, fv_sizes, fv_features, kf_mappoints, pairs, nnratio, check_ori,
                                       pair_params, uright, tri ? *tri : TriangulationDev{}, out_offsets, match_out,
                                       nmatches));
    ORBGPU_CUDA_TRY(cudaGetLastError());
    return ORBGPU_OK;
}

extern "C" int orbgpu_search_by_bow(const orbgpu_keypoint* kps, const uint8_t* desc, const int* offsets,
                                    const int* fv_counts, const int* fv_nodes, const int* fv_starts,
                                    const int* fv_sizes, const int* fv_features, const uint8_t* kf_mappoints,
                                    const int* pairs, int npairs, float nnratio, int check_ori,
                                    const int* out_offsets, int* match_out, int* nmatches, void* stream) {
    return search_by_bow(kps, desc, offsets, fv_counts, fv_nodes, fv_starts, fv_sizes, fv_features, kf_mappoints,
                         pairs, npairs, nnratio, check_ori, 0, out_offsets, match_out, nmatches, stream);
}

extern "C" int orbgpu_search_by_bow_keyframes(const orbgpu_keypoint* kps, const uint8_t* desc, const int* offsets,
                                              const int* fv_counts, const int* fv_nodes, const int* fv_starts,
                                              const int* fv_sizes, const int* fv_features,
                                              const uint8_t* kf_mappoints, const int* pairs, int npairs,
                                              float nnratio, int check_ori, const int* out_offsets, int* match_out,
                                              int* nmatches, void* stream) {
    return search_by_bow(kps, desc, offsets, fv_counts, fv_nodes, fv_starts, fv_sizes, fv_features, kf_mappoints,
                         pairs, npairs, nnratio, check_ori, 1, out_offsets, match_out, nmatches, stream);
}

extern "C" int orbgpu_vocabulary_create(int k, int L, int scoring, int weighting, int nnodes, const int* parents,
                                        const uint8_t* is_leaf, const uint8_t* descriptors, const double* weights,
                                        orbgpu_vocabulary** out) {
    if (!out || k < 0 || k > 20 || L < 1 || L > 10 || scoring < 0 || scoring > 5 || weighting < 0 || weighting > 3 ||
        nnodes < 1 || (nnodes > 1 && (!parents || !is_leaf || !descriptors || !weights))) {
        orbgpu_set_last_error("orbgpu_vocabulary_create: bad arguments", __FILE__, __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    *out = nullptr;
    const int nc = nnodes - 1;  // nodes after the root; node i + 1 is described by entry i
    std::vector<int> count(nnodes + 1, 0);
    for (int i = 0; i < nc; i++) {
        const int p = parents[i];
        if (p < 0 || p > i) {  // a parent must precede its child (the reference indexes m_nodes[pid])
            orbgpu_set_last_error("orbgpu_vocabulary_create: a node's parent does not precede it", __FILE__, __LINE__);
            return ORBGPU_ERR_BAD_ARG;
        }
        count[p + 1]++;
    }
    std::vector<int> start(nnodes + 1, 0);
    for (int p = 0; p < nnodes; p++) start[p + 1] = start[p] + count[p + 1];
    std::vector<int> fill(start.begin(), start.end() - 1), word(nnodes, 0);
    std::vector<int4> info(std::max(nc, 1));
    std::vector<uint8_t> cdesc((size_t)std::max(nc, 1) * 32);
    std::vector<double> w(nnodes, 0.0);
    int nwords = 0;
    for (int i = 0; i < nc; i++) {
        const int node = i + 1, pos = fill[parents[i]]++;
        info[pos] = make_int4(node, start[node], start[node + 1], 0);
        std::memcpy(&cdesc[(size_t)pos * 32], descriptors + (size_t)i * 32, 32);
        w[node] = weights[i];
        if (is_leaf[i]) word[node] = nwords++;
    }
    for (int4& c : info) c.w = word[c.x];
    orbgpu_vocabulary* v = new orbgpu_vocabulary();
    v->k = k;
    v->L = L;
    v->scoring = scoring;
    v->weighting = weighting;
    v->nnodes = nnodes;
    v->nwords = nwords;
    v->child_desc = nullptr;
    v->child_info = nullptr;
    v->root_end = start[1];
    v->node_weight = nullptr;
    cudaError_t e = cudaMalloc(&v->child_desc, cdesc.size());
    if (e == cudaSuccess) e = cudaMalloc(&v->child_info, sizeof(int4) * info.size());
    if (e == cudaSuccess) e = cudaMalloc(&v->node_weight, sizeof(double) * nnodes);
    if (e == cudaSuccess) e = cudaMemcpy(v->child_desc, cdesc.data(), cdesc.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(v->child_info, info.data(), sizeof(int4) * info.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(v->node_weight, w.data(), sizeof(double) * nnodes, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        orbgpu_vocabulary_destroy(v);
        orbgpu_set_last_error(cudaGetErrorString(e), __FILE__, __LINE__);
        return e == cudaErrorMemoryAllocation ? ORBGPU_ERR_OOM : ORBGPU_ERR_CUDA;
    }
    *out = v;
    return ORBGPU_OK;
}

extern "C" int orbgpu_vocabulary_load_text(const char* path, orbgpu_vocabulary** out) {
    // TemplatedVocabulary::loadFromTextFile (TemplatedVocabulary.h:1368-1460):
    // "k L scoring weighting", then "parent is_leaf d0 .. d31 weight" per node
    std::ifstream f(path ? path : "");
    std::string line;
    if (!out || !f.is_open() || !std::getline(f, line)) {
        orbgpu_set_last_error("orbgpu_vocabulary_load_text: cannot read the file", __FILE__, __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    int k = -1, L = -1, n1 = -1, n2 = -1;
    {
        std::stringstream hs(line);
        hs >> k >> L >> n1 >> n2;
    }
    std::vector<int> parents;
    std::vector<uint8_t> leaf, desc;
    std::vector<double> weights;
    while (std::getline(f, line)) {
        std::stringstream ls(line);
        int pid = -1, lf = 0;
        ls >> pid >> lf;
        uint8_t d[32];
        for (int i = 0; i < 32; i++) {
            int b = 0;
            ls >> b;
            d[i] = (uint8_t)b;
        }
        double w = 0;
        ls >> w;
        if (line.empty() || ls.fail()) {
            // an empty or short line: the reference appends a node whose
            // descriptor bytes are left unset
            orbgpu_set_last_error("orbgpu_vocabulary_load_text: malformed node line", __FILE__, __LINE__);
            return ORBGPU_ERR_BAD_ARG;
        }
        parents.push_back(pid);
        leaf.push_back(lf > 0 ? 1 : 0);
        desc.insert(desc.end(), d, d + 32);
        weights.push_back(w);
    }
    return orbgpu_vocabulary_create(k, L, n1, n2, (int)parents.size() + 1, parents.data(), leaf.data(), desc.data(),
                                    weights.data(), out);
}

extern "C" int orbgpu_vocabulary_destroy(orbgpu_vocabulary* v) {
    if (!v) return ORBGPU_OK;
    // transforms run on the caller's streams: all of them are done before the
    // tree is freed
    cudaDeviceSynchronize();
    cudaFree(v->child_desc);
    cudaFree(v->child_info);
    cudaFree(v->node_weight);
    delete v;
    return ORBGPU_OK;
}

extern "C" int orbgpu_vocabulary_size(const orbgpu_vocabulary* v, int* nwords, int* nnodes) {
    if (!v) return ORBGPU_ERR_BAD_ARG;
    if (nwords) *nwords = v->nwords;
    if (nnodes) *nnodes = v->nnodes;
    return ORBGPU_OK;
}

extern "C" int orbgpu_bow_transform(const orbgpu_vocabulary* v, const uint8_t* desc, const int* offsets, int nframes,
                                    int levelsup, int* word_ids, double* weights, int* node_ids, int* bow_counts,
                                    int* bow_words, double* bow_values, int* fv_counts, int* fv_nodes, int* fv_starts,
                                    int* fv_sizes, int* fv_features, void* stream) {
    if (!v || nframes < 0 ||
        (nframes > 0 && (!desc || !offsets || !word_ids || !weights || !node_ids || !bow_counts || !bow_words ||
                         !bow_values || !fv_counts || !fv_nodes || !fv_starts || !fv_sizes || !fv_features)) ||
        ((uintptr_t)desc & 15)) {
        orbgpu_set_last_error("orbgpu_bow_transform: bad arguments", __FILE__, __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    if (nframes == 0) return ORBGPU_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (v->nwords == 0) {
        // TemplatedVocabulary::transform returns empty vectors for an empty vocabulary
        ORBGPU_CUDA_TRY(cudaMemsetAsync(bow_counts, 0, sizeof(int) * nframes, st));
        ORBGPU_CUDA_TRY(cudaMemsetAsync(fv_counts, 0, sizeof(int) * nframes, st));
        return ORBGPU_OK;
    }
    ORBGPU_CUDA_TRY(allow_max_dynamic_smem(k_bow_assemble));
    const int blocks = nsm_of_current_device() * 8;
    k_bow_descend<<<blocks, BOW_THREADS, 0, st>>>(reinterpret_cast<const uint4*>(desc), offsets, nframes,
                                                  v->child_desc, v->child_info, v->root_end, v->node_weight,
                                                  v->L - levelsup, word_ids, weights, node_ids);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    k_bow_assemble<<<2 * nframes, BOW_ASM_THREADS, BOW_MAX_FEATURES * 8, st>>>(
        offsets, word_ids, weights, node_ids, v->weighting, v->scoring, bow_counts, bow_words, bow_values, fv_counts,
        fv_nodes, fv_starts, fv_sizes, fv_features);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    return ORBGPU_OK;
}

extern "C" int orbgpu_triangulation_epipole(const float* Cw1, const float* T2, const float* K2, float* ex,
                                            float* ey) {
    if (!Cw1 || !T2 || !K2 || !ex || !ey) return ORBGPU_ERR_BAD_ARG;
    // C2 = R2w * Cw + t2w (src/ORBmatcher.cc:897-901): the 3 x 3 product
    // accumulated in double and rounded to float, then a float add
    float C2[3];
    for (int r = 0; r < 3; r++) {
        double s = 0.0;
        for (int k = 0; k < 3; k++) s += (double)T2[4 * r + k] * (double)Cw1[k];
        C2[r] = (float)s + T2[4 * r + 3];
    }
    const float invz = 1.0f / C2[2];
    *ex = K2[0] * C2[0] * invz + K2[2];
    *ey = K2[1] * C2[1] * invz + K2[3];
    return ORBGPU_OK;
}

extern "C" int orbgpu_search_for_triangulation(const orbgpu_keypoint* kps, const uint8_t* desc, const int* offsets,
                                               const int* fv_counts, const int* fv_nodes, const int* fv_starts,
                                               const int* fv_sizes, const int* fv_features,
                                               const uint8_t* has_mappoint, const float* uright, const int* pairs,
                                               int npairs, const float* pair_params, const float* scale_factors,
                                               const float* level_sigma2, int nlevels, int only_stereo,
                                               int check_ori, const int* out_offsets, int* match_out,
                                               int* nmatches, void* stream) {
    if (!uright || (npairs > 0 && !pair_params) || !scale_factors || !level_sigma2 || nlevels < 1 || nlevels > 16) {
        orbgpu_set_last_error("orbgpu_search_for_triangulation: bad arguments", __FILE__, __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    TriangulationDev tri;
    std::memset(&tri, 0, sizeof(tri));
    for (int l = 0; l < nlevels; l++) {
        tri.scale[l] = scale_factors[l];
        tri.sigma2[l] = level_sigma2[l];
    }
    // octaves past nlevels read the reference's vectors out of range: they are rejected here
    for (int l = nlevels; l < 16; l++) tri.scale[l] = tri.sigma2[l] = 0.0f;
    tri.only_stereo = only_stereo ? 1 : 0;
    return search_by_bow(kps, desc, offsets, fv_counts, fv_nodes, fv_starts, fv_sizes, fv_features, has_mappoint,
                         pairs, npairs, 0.0f, check_ori, 2, out_offsets, match_out, nmatches, stream, pair_params,
                         uright, &tri);
}
