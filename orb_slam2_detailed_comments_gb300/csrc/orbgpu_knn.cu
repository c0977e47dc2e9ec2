// orbgpu_knn.cu -- brute-force k = 2 Hamming nearest neighbours.
//
// Popcount path: every thread owns one query (its 256 bits in registers); the
// warps of a block share 32 queries and split each tile of train rows between
// them through shared memory; the train set is split into slices across
// blocks so the grid covers the GPU, and a merge kernel combines the
// per-slice (best, second) pairs.  Ties go to the lower train index, the rule
// of a sequential scan over DescriptorDistance (src/ORBmatcher.cc:2083-2103).
#include <algorithm>
#include <mutex>

#include "orbgpu_host.h"

cudaStream_t orbgpu_matcher_stream_internal(orbgpu_matcher* m);

namespace orbgpu {

#define KNN_Q 32       // queries per block, one per lane
#define KNN_WARPS 8    // warps per block, each with its share of a tile
#define KNN_TILE 256   // train rows per tile (a slice is a whole number of tiles)
#define KNN_SHARE (KNN_TILE / KNN_WARPS)

// Full adder of three bit planes.
__device__ __forceinline__ void knn_full_add(uint32_t a, uint32_t b, uint32_t c, uint32_t& sum, uint32_t& carry) {
    sum = a ^ b ^ c;
    carry = (a & b) | (c & (a | b));
}
// hamming256 with four population counts instead of eight: full adders reduce
// the eight XOR words to planes of weight 1, 1, 2 and 4 (Harley and Seal).
// POPC issues at a quarter of the rate of the logic operations, and this
// loop does nothing else.
__device__ __forceinline__ uint32_t knn_hamming(const uint4 a0, const uint4 a1, const uint4 b0, const uint4 b1) {
    uint32_t s1, c1, s2, c2, s3, c3, t, f;
    knn_full_add(a0.x ^ b0.x, a0.y ^ b0.y, a0.z ^ b0.z, s1, c1);
    knn_full_add(a0.w ^ b0.w, a1.x ^ b1.x, a1.y ^ b1.y, s2, c2);
    knn_full_add(s1, s2, a1.z ^ b1.z, s3, c3);
    knn_full_add(c1, c2, c3, t, f);
    return __popc(s3) + __popc(a1.w ^ b1.w) + 2 * __popc(t) + 4 * __popc(f);
}

// (b1, b2), the two smallest keys so far, with another pair o1 <= o2.
__device__ __forceinline__ void knn_merge_pair(unsigned long long& b1, unsigned long long& b2, unsigned long long o1,
                                               unsigned long long o2) {
    const unsigned long long hi = max(b1, o1);
    b1 = min(b1, o1);
    b2 = min(min(b2, o2), hi);
}

// Bound by issue and POPC together: 13.3 ms at 50,000 x 200,000 (25 thread
// instructions a pair), 18.1 with eight POPC a pair and a branch per improved
// row.  Eight warps share a block's 32 queries so that 2,000 x 2,000 fills the
// SMs (504 blocks; 128 queries a block were 128): 10 us instead of 17.
//
// Keys pack (distance << 23 | row), so a (distance, index) top-2 is three
// min/max operations per row; rows count from the start of a run of KNN_RUN,
// after which the two keys move to 64 bits (distance << 32 | train index).
#define KNN_RUN (1 << 22)  // rows, a whole number of tiles
__global__ void __launch_bounds__(32 * KNN_WARPS) k_knn_popc(const uint4* __restrict__ q, int nq,
                                                             const uint4* __restrict__ t, int nt, int slice,
                                                             int4* __restrict__ partial) {
    __shared__ uint4 tile[KNN_TILE * 2];
    __shared__ ulonglong2 s_best[KNN_WARPS][KNN_Q];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int qi = blockIdx.x * KNN_Q + lane;
    const long long t0 = (long long)blockIdx.y * slice, t1 = min((long long)nt, t0 + slice);
    uint4 a0 = make_uint4(0, 0, 0, 0), a1 = a0;
    if (qi < nq) {
        a0 = q[2 * (size_t)qi];
        a1 = q[2 * (size_t)qi + 1];
    }
    constexpr unsigned long long NONE = 0x7fffffffffffffffull;  // distance 0x7fffffff, index -1
    unsigned long long b1 = NONE, b2 = NONE;
    for (long long r0 = t0; r0 < t1; r0 += KNN_RUN) {
        const int rows = (int)min((long long)KNN_RUN, t1 - r0);
        uint32_t k1 = 0xFFFFFFFFu, k2 = 0xFFFFFFFFu;
        for (int base = 0; base < rows; base += KNN_TILE) {
            const int nb = min(KNN_TILE, rows - base);
            __syncthreads();
            for (int k = threadIdx.x; k < 2 * nb; k += 32 * KNN_WARPS) tile[k] = t[2 * (size_t)(r0 + base) + k];
            __syncthreads();
            const int j0 = warp * KNN_SHARE, j1 = min(nb, j0 + KNN_SHARE);
#pragma unroll 4
            for (int j = j0; j < j1; j++) {
                const uint32_t key = (knn_hamming(a0, a1, tile[2 * j], tile[2 * j + 1]) << 23) | (uint32_t)(base + j);
                const uint32_t hi = max(k1, key);
                k1 = min(k1, key);
                k2 = min(k2, hi);
            }
        }
        auto wide = [&](uint32_t k) {
            return k == 0xFFFFFFFFu ? NONE : ((unsigned long long)(k >> 23) << 32) | (unsigned long long)(r0 + (k & 0x7FFFFF));
        };
        knn_merge_pair(b1, b2, wide(k1), wide(k2));
    }
    s_best[warp][lane] = make_ulonglong2(b1, b2);
    __syncthreads();
    if (warp == 0 && qi < nq) {
#pragma unroll
        for (int w = 1; w < KNN_WARPS; w++) knn_merge_pair(b1, b2, s_best[w][lane].x, s_best[w][lane].y);
        partial[(size_t)blockIdx.y * nq + qi] =
            make_int4((int)(uint32_t)b1, (int)(b1 >> 32), (int)(uint32_t)b2, (int)(b2 >> 32));
    }
}

// Slices of the train set for nq queries: about eight blocks per SM, each
// slice a whole number of tiles, at most max_slices of them.
static void knn_slices(int nq, int nt, int max_slices, int* slice, int* nslices) {
    const int qblocks = (nq + KNN_Q - 1) / KNN_Q, tiles = std::max(1, nt / KNN_TILE + (nt % KNN_TILE != 0));
    int n = std::max(1, std::min(tiles, (8 * nsm_of_current_device() + qblocks - 1) / qblocks));
    n = std::min(n, std::max(1, max_slices));
    const int per = (tiles + n - 1) / n;  // tiles of a slice
    *slice = per <= 0x7fffffff / KNN_TILE ? per * KNN_TILE : 0x7fffffff;
    *nslices = (tiles + per - 1) / per;
}

__global__ void k_knn_merge(const int4* __restrict__ partial, int nq, int nslices, int* idx1, int* d1, int* idx2,
                            int* d2) {
    const int qi = blockIdx.x * blockDim.x + threadIdx.x;
    if (qi >= nq) return;
    // slices are in increasing train order, so strict comparisons keep the
    // lower index on ties
    int b1 = 0x7fffffff, b2 = 0x7fffffff, i1 = -1, i2 = -1;
    for (int s = 0; s < nslices; s++) {
        const int4 p = partial[(size_t)s * nq + qi];
        if (p.x >= 0) {
            if (p.y < b1) {
                b2 = b1; i2 = i1; b1 = p.y; i1 = p.x;
            } else if (p.y < b2) {
                b2 = p.y; i2 = p.x;
            }
        }
        if (p.z >= 0) {
            if (p.w < b1) {
                b2 = b1; i2 = i1; b1 = p.w; i1 = p.z;
            } else if (p.w < b2) {
                b2 = p.w; i2 = p.z;
            }
        }
    }
    idx1[qi] = i1;
    d1[qi] = b1;
    idx2[qi] = i2;
    d2[qi] = b2;
}

// Lowe's ratio test in the reference's form (src/ORBmatcher.cc:647:
// bestDist < (float)bestDist2 * nnratio); no second neighbour rejects.
__global__ void k_knn_accept(const int* d1, const int* d2, int n, float ratio, uint8_t* accept) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = d1[i], s = d2[i];
    accept[i] = (s != 0x7fffffff && (float)b < __fmul_rn((float)s, ratio)) ? 1 : 0;
}

}  // namespace orbgpu

using namespace orbgpu;

extern "C" int orbgpu_knn2_accept(const int* d1, const int* d2, int n, float ratio, uint8_t* accept, void* stream) {
    if (n < 0 || (n > 0 && (!d1 || !d2 || !accept))) return ORBGPU_ERR_BAD_ARG;
    if (n == 0) return ORBGPU_OK;
    cudaStream_t st = (cudaStream_t)stream;
    k_knn_accept<<<(n + 255) / 256, 256, 0, st>>>(d1, d2, n, ratio, accept);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    ORBGPU_CUDA_TRY(cudaStreamSynchronize(st));
    return ORBGPU_OK;
}

int orbgpu_knn2_tc(orbgpu_matcher* m, const uint8_t* query, int nq, const uint8_t* train, int nt, int* idx1, int* d1,
                   int* idx2, int* d2);

// The automatic choice: the tensor cores from the tuned number of pairs on, but
// not where their operands (128 bytes a row, of a query pair and a train tile
// at least) cost more than the pairs.  A call in microseconds, popcount against
// tensor cores:
// * up to 256 train rows: 1,000,000 x 16 119 / 339, x 128 242 / 365, x 256 394 /
//   372; 64,000 x 256 72 / 77, x 512 93 / 81;
// * under 128 queries, a train set whose operands a matcher does not keep:
//   8 x 8,000,000 722 / 1,382, 64 898 / 1,384, 128 1,457 / 1,381; kept, 8 x
//   4,000,000 488 / 281.
extern "C" int orbgpu_debug_knn_algo(int nq, int nt) {
    if (nt >= (1 << 23)) return 0;  // the tensor-core epilogue packs train indices in 23 bits
    if ((long long)nq * nt < tunables().knn_tc_min_pairs || nt <= 256) return 0;
    return nq >= 128 || (size_t)nt * 128 <= KNN_KEEP_BYTES;
}

extern "C" int orbgpu_knn2(orbgpu_matcher* m, const uint8_t* query, int nq, const uint8_t* train, int nt, int* idx1,
                           int* d1, int* idx2, int* d2, int algo) {
    if (!m || nq < 0 || nt < 0 || (nq > 0 && (!query || !idx1 || !d1 || !idx2 || !d2)) || (nt > 0 && !train) ||
        (algo != 0 && algo != 1 && algo != -1))
        return ORBGPU_ERR_BAD_ARG;
    if (nq == 0) return ORBGPU_OK;
    if (algo == -1) algo = orbgpu_debug_knn_algo(nq, nt);
    if (nt >= (1 << 23)) algo = 0;
    if (algo == 1 && nt > 0) return orbgpu_knn2_tc(m, query, nq, train, nt, idx1, d1, idx2, d2);
    cudaStream_t st = orbgpu_matcher_stream_internal(m);
    int slice, nslices;
    knn_slices(nq, nt, 0x7fffffff, &slice, &nslices);
    KnnWorkspace work(m);
    const int rc = work.take(sizeof(int4) * (size_t)nq * nslices);
    if (rc != ORBGPU_OK) return rc;
    int4* partial = (int4*)work.data();
    dim3 grid((nq + KNN_Q - 1) / KNN_Q, nslices);
    k_knn_popc<<<grid, 32 * KNN_WARPS, 0, st>>>((const uint4*)query, nq, (const uint4*)train, nt, slice, partial);
    k_knn_merge<<<(nq + 255) / 256, 256, 0, st>>>(partial, nq, nslices, idx1, d1, idx2, d2);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    ORBGPU_CUDA_TRY(cudaStreamSynchronize(st));
    return ORBGPU_OK;
}

// ---------------------------------------------------------------- allocation-free variant
// orbgpu_knn2_noalloc keeps its per-slice (best, second) pairs in this
// file-scope device array instead of memory it allocates.  Each GPU that
// loads the library holds the array (16 MiB) until the process exits.
#define ORBGPU_KNN_NOALLOC_MAX_PARTIAL (1 << 20)
static __device__ __align__(256) int4 g_knn_noalloc_partial[ORBGPU_KNN_NOALLOC_MAX_PARTIAL];

namespace {
std::mutex g_noalloc_mutex;
// device address of the array, per device ordinal, looked up once; a
// cudaDeviceReset ends the context that address belongs to, so it must not be
// followed by further calls in the same process
int4* g_noalloc_partial[256] = {};
}  // namespace

extern "C" int orbgpu_knn2_noalloc(const uint8_t* query, int nq, const uint8_t* train, int nt, int* idx1, int* d1,
                                   int* idx2, int* d2, void* stream) {
    if (nq < 0 || nt < 0 || (nq > 0 && (!query || !idx1 || !d1 || !idx2 || !d2)) || (nt > 0 && !train)) {
        orbgpu_set_last_error("invalid kNN arguments", __FILE__, __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    if (nq > ORBGPU_KNN_NOALLOC_MAX_PARTIAL) {
        orbgpu_set_last_error("orbgpu_knn2_noalloc: more than 1048576 query rows (its fixed scratch holds one "
                              "(best, second) pair per query per train slice)", __FILE__, __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    if (nq == 0) return ORBGPU_OK;
    int dev = 0;
    ORBGPU_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 256) {
        orbgpu_set_last_error("orbgpu_knn2_noalloc: device ordinal beyond 255", __FILE__, __LINE__);
        return ORBGPU_ERR_BAD_ARG;
    }
    int4* partial = nullptr;
    {
        // first call on a device: look up the array's device address with
        // that device current (the host-side symbol is not a device address)
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_partial[dev]) {
            void* p = nullptr;
            ORBGPU_CUDA_TRY(cudaGetSymbolAddress(&p, g_knn_noalloc_partial));
            g_noalloc_partial[dev] = (int4*)p;
        }
        partial = g_noalloc_partial[dev];
    }
    cudaStream_t st = (cudaStream_t)stream;
    int slice, nslices;
    knn_slices(nq, nt, ORBGPU_KNN_NOALLOC_MAX_PARTIAL / nq, &slice, &nslices);
    // every partial entry read by the merge is written by the popcount
    // kernel of the same call, so nothing is cleared between calls
    dim3 grid((nq + KNN_Q - 1) / KNN_Q, nslices);
    k_knn_popc<<<grid, 32 * KNN_WARPS, 0, st>>>((const uint4*)query, nq, (const uint4*)train, nt, slice, partial);
    k_knn_merge<<<(nq + 255) / 256, 256, 0, st>>>(partial, nq, nslices, idx1, d1, idx2, d2);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    return ORBGPU_OK;
}
