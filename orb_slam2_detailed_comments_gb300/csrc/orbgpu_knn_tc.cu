// orbgpu_knn_tc.cu -- brute-force k = 2 Hamming kNN on the 5th-generation
// tensor cores (tcgen05).
//
// Each 256-bit descriptor is expanded to 256 FP4 (E2M1) values, +1 for a 0
// bit and -1 for a 1 bit, two to a byte.  With all block scales 1 the dot
// product of two expansions is 256 - 2 * Hamming, exact in the FP32
// accumulator, so
//     Hamming = (256 - dot) / 2.
// The expansions are written in the tensor cores' shared-memory operand
// layout (K-major, no swizzle: 8-row x 16-byte core matrices, 128 bytes
// each, the 8 core matrices of one 8-row group back to back), so a 128-row
// query tile (16 KiB) and a 160-row train tile (20 KiB) are single
// contiguous bulk copies.
//
// Work items are (two query tiles, train tile) in query-major order, dealt to
// one CTA per SM as equal contiguous runs.  For each of the two query tiles an
// elected thread issues 4 MMAs (M=128, N=160, K=64) into a TMEM accumulator
// (128 lanes x 160 FP32 columns, one for each of three issuing warps; the
// block scales take the last 32 columns), commits them to an mbarrier, and the
// accumulator's four epilogue warps (one per TMEM lane quadrant, a thread per
// query) read the largest dot product of every 32 train rows with
// tcgen05.ld.red; train tiles run through six shared-memory buffers.  All waits are bounded: on timeout
// the CTA records an error flag, drains, frees its TMEM and returns.
//
// A thread keeps its query's two best groups of 32 train rows, ordered by
// (least distance in the group, group index).  The query's two nearest rows
// lie in these two groups: the nearest is the first least of the best group
// (groups are consecutive index ranges, so the lower index of equal distances
// is in the lower group), and the second is either another row of that group
// or the first least of the next best group.  k_knn_tc_finish reads the 64
// rows' descriptors again and picks the two.  (Keeping the two best rows
// themselves in the epilogue took a branch wherever a row of a warp improved,
// in most tiles: 1.05 ms instead of 0.73 at 50,000 x 200,000.)
#include <algorithm>
#include <cstdio>
#include <mutex>

#include "orbgpu_async.cuh"
#include "orbgpu_host.h"

cudaStream_t orbgpu_matcher_stream_internal(orbgpu_matcher* m);

namespace orbgpu {

// the FP8 operand layout's test: one 128 x 256 tile of +-1 rows
#define TCP_M 128
#define TCP_N 256
#define TCP_K 256                        // bytes (= FP8 elements) per row
#define TCP_QTILE_BYTES (TCP_M * TCP_K)  // 32 KiB
#define TCP_TTILE_BYTES (TCP_N * TCP_K)  // 64 KiB

// the kNN kernel.  N = 160: three accumulators of 160 columns leave the 32
// TMEM columns that hold the block scales.
#define TC_M 128
#define TC_N 160
#define TC_ROW 128                      // bytes per row (256 FP4 elements)
#define TC_QTILE_BYTES (TC_M * TC_ROW)  // 16 KiB
#define TC_QPAIR 2                      // query tiles that share each train tile
#define TC_Q (TC_QPAIR * TC_M)          // their queries
#define TC_QPAIR_BYTES (TC_QPAIR * TC_QTILE_BYTES)
#define TC_TTILE_BYTES (TC_N * TC_ROW)  // 20 KiB
#define TC_STAGES 6                     // train tiles in shared memory
#define TC_ACCS 3                       // accumulators, each with an issuing warp and four epilogue warps
#define TC_SCALE_COL (TC_ACCS * TC_N)   // first TMEM column of the scales
#define TC_EPI_WARPS (4 * TC_ACCS)      // a warp per accumulator and TMEM lane quadrant
#define TC_GROUP 32                     // train rows of a group
#define TC_GROUPS (TC_N / TC_GROUP)     // groups of a train tile
#define TC_THREADS (32 * (TC_EPI_WARPS + 1 + TC_ACCS))  // + producer warp + MMA warps
static_assert(TC_N % TC_GROUP == 0, "whole groups");
// An issuer takes tiles of two items in three.  With the stages a multiple of
// the accumulators it takes from a stage either at every fill or never, so it
// sees every phase of the stage's barrier and a parity names one fill.
static_assert(TC_STAGES % TC_ACCS == 0, "an issuer would skip fills of a stage");

// ---------------------------------------------------------------- operand layout
// Byte offset of byte k of row r inside a tile of 256-byte rows (the
// self-test's) stored K-major without swizzle: core matrix (r / 8, k / 16) is
// 128 contiguous bytes (8 rows of 16 bytes); the 16 core matrices along K of
// one 8-row group are consecutive (leading-dimension stride 128 B), 8-row
// groups are 2048 B apart (stride dimension).  The kNN kernel's 128-byte rows
// follow the same scheme with 8 core matrices and 1024 B.
__host__ __device__ __forceinline__ uint32_t tc_offset(int r, int k) {
    return (uint32_t)((r >> 3) * 2048 + (k >> 4) * 128 + (r & 7) * 16 + (k & 15));
}

// Expands n descriptors (32 bytes) into tiled FP8 +-1 rows; rows past n are
// +1 everywhere (their distances are discarded by the index bound).  One
// thread per 16 bits: the 16 FP8 values of one core-matrix row, one 16-byte
// store.
__global__ void k_expand_fp8(const uint8_t* __restrict__ desc, int n, int tile_rows, uint8_t* __restrict__ out) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int row = (int)(t >> 4), c = (int)(t & 15);  // bits 16c .. 16c + 15 of the row
    const int tile = row / tile_rows, r = row - tile * tile_rows;
    uint32_t bits = 0;
    if (row < n) bits = (uint32_t)desc[(size_t)row * 32 + 2 * c] | ((uint32_t)desc[(size_t)row * 32 + 2 * c + 1] << 8);
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        uint32_t v = 0;
#pragma unroll
        for (int b = 0; b < 4; b++) v |= (((bits >> (4 * q + b)) & 1u) ? 0xB8u : 0x38u) << (8 * b);  // 1 bit -> -1.0
        w[q] = v;
    }
    *reinterpret_cast<uint4*>(out + (size_t)tile * tile_rows * TCP_K + tc_offset(r, 16 * c)) = make_uint4(w[0], w[1], w[2], w[3]);
}

// A word at any address.
__device__ __forceinline__ uint32_t load_u32(const uint8_t* p) {
    if (((uintptr_t)p & 3) == 0) return *reinterpret_cast<const uint32_t*>(p);
    return (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
}

// Expands the nq query and nt train descriptors (32 bytes each) into their
// tiles of FP4 +-1 rows; rows past the end repeat the last row (the largest
// dot product of a group that holds some real rows stays that of a real row).
// One thread per 32 bits: the 32 FP4
// values of one core-matrix row, one 16-byte store, in the order of the
// output (thread t of a set writes bytes [16 t, 16 t + 16) of its tiles, whose
// 8-row groups are contiguous across tiles).  Also clears the status word.
__global__ void __launch_bounds__(256) k_expand_fp4(const uint8_t* __restrict__ q, int nq, long q_threads,
                                                    uint8_t* __restrict__ q_out, const uint8_t* __restrict__ t, int nt,
                                                    long t_threads, uint8_t* __restrict__ t_out, int* status) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *status = 0;
    const uint8_t* src = q;
    uint8_t* dst = q_out;
    int n = nq;
    if (i >= q_threads) {
        i -= q_threads;
        if (i >= t_threads) return;
        src = t;
        dst = t_out;
        n = nt;
    }
    const long row = min((i >> 6) * 8 + (i & 7), (long)n - 1);
    const int c = (int)(i >> 3) & 7;  // bits 32c .. 32c + 31 of the row
    const uint32_t bits = load_u32(src + row * 32 + 4 * c);
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        uint32_t v = (bits >> (8 * k)) & 0xFFu;  // bit b to bit 4 b + 3: the sign of nibble b
        v = (v | (v << 12)) & 0x000F000Fu;
        v = (v | (v << 6)) & 0x03030303u;
        v = (v | (v << 3)) & 0x11111111u;
        w[k] = 0x22222222u | (v << 3);  // E2M1: 0x2 is 1.0, 0xA is -1.0
    }
    *reinterpret_cast<uint4*>(dst + 16 * i) = make_uint4(w[0], w[1], w[2], w[3]);
}

// ---------------------------------------------------------------- PTX wrappers
// K-major, no swizzle shared-memory operand descriptor.
__device__ __forceinline__ uint64_t smem_desc(const void* base, uint32_t lbo, uint32_t sbo) {
    const uint64_t a = (uint64_t)((smem_u32(base) >> 4) & 0x3FFF);
    return a | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f8f6f4: D = FP32, A = B = E4M3, both K-major.
__host__ __device__ __forceinline__ uint32_t idesc_e4m3(int M, int N) {
    return (1u << 4)                   // D format F32
           | (0u << 7) | (0u << 10)    // A, B format E4M3
           | ((uint32_t)(N >> 3) << 17)
           | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum));
}
// Instruction descriptor of kind::mxf4: A = B = E2M1, both K-major, block
// scales UE8M0 (scale ids 0), D = FP32, K = 64.
__host__ __device__ __forceinline__ uint32_t idesc_mxf4(int M, int N) {
    return (1u << 7) | (1u << 10)  // A, B format E2M1
           | ((uint32_t)(N >> 3) << 17)
           | (1u << 23)  // scales UE8M0
           | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tc_mma_mxf4(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t scale_tmem, int accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%5], p;\n\t}" ::"r"(
            dtmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum), "r"(scale_tmem));
}
// One lane of the (converged) warp.
__device__ __forceinline__ bool tc_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Each lane's largest of 32 consecutive FP32 columns of this warp's 32 TMEM
// lanes, reduced on the way to the registers (without the wait; the columns
// themselves land in r).
__device__ __forceinline__ float tc_max32(uint32_t taddr, uint32_t* r) {
    float m;
    asm volatile(
        "tcgen05.ld.red.sync.aligned.32x32b.x32.max.f32 {"
        "%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%2"
        "7,%28,%29,%30,%31"
        "}, %32, [%33];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=f"(m)
        : "r"(taddr));
    return m;
}
// The same word into 8 consecutive columns of this warp's 32 TMEM lanes.
__device__ __forceinline__ void tc_fill8(uint32_t taddr, uint32_t v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr), "r"(v) : "memory");
}

// Block scales of 1 (UE8M0 0x7F) in the scale columns of this warp's 32 TMEM
// lanes (ta: its first lane); every lane holds them, whichever an MMA reads.
__device__ __forceinline__ void tc_fill_scales(uint32_t ta) {
    for (int c = 0; c < 512 - TC_SCALE_COL; c += 8) tc_fill8(ta + TC_SCALE_COL + c, 0x7F7F7F7Fu);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// A tile's operand descriptor, and the MMAs of two tiles' whole rows.
__device__ __forceinline__ uint64_t tc_operand(const void* tile) { return smem_desc(tile, 128, 8 * TC_ROW); }
__device__ __forceinline__ void tc_tile_mma(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t scales) {
#pragma unroll
    for (int ks = 0; ks < TC_ROW / 32; ks++) tc_mma_mxf4(d, ad + 16 * ks, bd + 16 * ks, idesc, scales, ks > 0);
}

// 32 consecutive FP32 columns of this warp's 32 TMEM lanes.
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// ---------------------------------------------------------------- probe
// One MMA group of a 128 x 256 tile over K = 256: D[i][j] = sum_k A[i][k] B[j][k]
// written to out (128 x 256 floats), for the layout self-test.
__global__ void __launch_bounds__(128) k_tc_probe(const uint8_t* qa, const uint8_t* tb, float* out, int* status, uint32_t lbo,
                                                  uint32_t sbo) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    uint8_t* sA = tc_smem;
    uint8_t* sB = tc_smem + TCP_QTILE_BYTES;
    __shared__ __align__(8) uint64_t bar_load, bar_mma;
    __shared__ uint32_t tmem_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(&bar_load, 1);
        mbar_init(&bar_mma, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(&tmem_base)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    bool ok = true;
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar_load, TCP_QTILE_BYTES + TCP_TTILE_BYTES);
        bulk_g2s(sA, qa, TCP_QTILE_BYTES, &bar_load);
        bulk_g2s(sB, tb, TCP_TTILE_BYTES, &bar_load);
        ok = mbar_wait(&bar_load, 0);
        if (ok) {
            tc_fence_after();
            const uint32_t idesc = idesc_e4m3(TCP_M, TCP_N);
            for (int ks = 0; ks < TCP_K / 32; ks++) {
                const uint64_t ad = smem_desc(sA + ks * 256, lbo, sbo);
                const uint64_t bd = smem_desc(sB + ks * 256, lbo, sbo);
                tc_mma(tmem, ad, bd, idesc, ks > 0);
            }
            tc_commit(&bar_mma);
        }
        if (!ok) {
            atomicOr(status, 1);
            mbar_wait(&bar_load, 0);  // give the copies in flight one more bounded wait
        }
    }
    __syncthreads();
    if (!(*status & 1)) {
        const bool done = mbar_wait(&bar_mma, 0);
        if (!done && lane == 0) atomicOr(status, 2);
        tc_fence_after();
        if (done) {
            const int row = warp * 32 + lane;
            for (int c = 0; c < TCP_N; c += 32) {
                float v[32];
                tc_ld32(tmem + ((uint32_t)(warp * 32) << 16) + c, v);
                for (int i = 0; i < 32; i++) out[(size_t)row * TCP_N + c + i] = v[i];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem));
}

// One query tile against one train tile as k_knn_tc takes them (operand strides,
// instruction descriptor, scale columns, the reduction of a group's columns):
// the 128 x 160 dot products and every row's five group maxima.
__global__ void __launch_bounds__(128) k_knn_tile_probe(const uint8_t* qa, const uint8_t* tb, float* dots, float* maxima,
                                                        int* status) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    uint8_t* sB = tc_smem + TC_QTILE_BYTES;
    __shared__ __align__(8) uint64_t bar_load, bar_mma;
    __shared__ uint32_t tmem_base;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        mbar_init(&bar_load, 1);
        mbar_init(&bar_mma, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base, ta = tmem + ((uint32_t)(warp * 32) << 16);
    tc_fill_scales(ta);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar_load, TC_QTILE_BYTES + TC_TTILE_BYTES);
        bulk_g2s(tc_smem, qa, TC_QTILE_BYTES, &bar_load);
        bulk_g2s(sB, tb, TC_TTILE_BYTES, &bar_load);
        if (mbar_wait(&bar_load, 0)) {
            tc_fence_after();
            tc_tile_mma(tmem, tc_operand(tc_smem), tc_operand(sB), idesc_mxf4(TC_M, TC_N), tmem + TC_SCALE_COL);
            tc_commit(&bar_mma);
        } else {
            atomicOr(status, 1);
            mbar_wait(&bar_load, 0);  // give the copies in flight one more bounded wait
        }
    }
    __syncthreads();
    if (!(*status & 1)) {
        const bool done = __all_sync(0xffffffffu, mbar_wait(&bar_mma, 0));
        if (!done) atomicOr(status, 2);
        tc_fence_after();
        for (int g = 0; done && g < TC_GROUPS; g++) {
            float v[32];
            uint32_t r[TC_GROUP];
            tc_ld32(ta + (uint32_t)(g * TC_GROUP), v);
            const float m = tc_max32(ta + (uint32_t)(g * TC_GROUP), r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            for (int i = 0; i < TC_GROUP; i++) dots[(size_t)threadIdx.x * TC_N + g * TC_GROUP + i] = v[i];
            maxima[threadIdx.x * TC_GROUPS + g] = m;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// mbar_wait_sleep by every lane of the warp, with one outcome.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_wait_sleep(bar, parity));
}

// ---------------------------------------------------------------- kNN kernel
// qa: query tiles of 16 KiB in pairs, tb: train tiles (tt of 20 KiB).  CTA b
// takes items [b run, (b + 1) run) of the (query pair, train tile) items in
// query-major order: every SM has the same number of tiles to within one,
// whatever the sizes (a grid of query tiles left the last of 2.6 waves half
// empty at 50,000 queries).  The items of one query pair that fall to a CTA
// are a segment; its per-query best two groups go to slot (CTA - first CTA of
// that pair) of 'partial'.
// What bounds it (50,000 x 200,000, 0.73 ms; FP8 operands with a grid of query
// tiles took 1.76 ms): a query tile's four MMAs take about 340 cycles of the
// tensor core, which is busy 71 % of the time (0.52 ms); the rest is the round
// trip between MMA, epilogue and the accumulator's release that three
// accumulators do not quite cover.  Two query tiles share a train tile
// because one bulk copy of 20 KiB takes its warp longer than 340 cycles.
struct TcItem {
    int q, t;  // query pair, train tile
};
__global__ void __launch_bounds__(TC_THREADS, 1)
    k_knn_tc(const uint8_t* __restrict__ qa, const uint8_t* __restrict__ tb, int nq, int nt, long items, int tt, int run,
             uint2* __restrict__ partial, int* status) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    uint8_t* sA = tc_smem;                       // two query pairs
    uint8_t* sB = tc_smem + 2 * TC_QPAIR_BYTES;  // TC_STAGES train tiles
    __shared__ __align__(8) uint64_t bar_a[2], bar_a_free[2], bar_full[TC_STAGES], bar_empty[TC_STAGES],
        bar_acc[TC_ACCS], bar_acc_free[TC_ACCS];
    __shared__ uint32_t tmem_base;
    __shared__ uint2 s_part[TC_ACCS][TC_Q];
    // the warp's role as a uniform value: the MMA's descriptors then live in
    // uniform registers
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int producer = TC_EPI_WARPS, issuer = TC_EPI_WARPS + 1;  // issuers: issuer .. issuer + TC_ACCS - 1
    const long i0 = (long)blockIdx.x * run;
    const int nitem = (int)max(0L, min((long)run, items - i0));
    const TcItem first{(int)(i0 / tt), (int)(i0 % tt)};
    auto next = [&](TcItem& it) {
        if (++it.t == tt) {
            it.t = 0;
            it.q++;
        }
    };
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; i++) {
            mbar_init(&bar_a[i], 1);
            mbar_init(&bar_a_free[i], TC_ACCS);
        }
        for (int i = 0; i < TC_ACCS; i++) {
            mbar_init(&bar_acc[i], 1);
            mbar_init(&bar_acc_free[i], 4);
        }
        for (int i = 0; i < TC_STAGES; i++) {
            mbar_init(&bar_full[i], 1);
            mbar_init(&bar_empty[i], TC_QPAIR);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == issuer) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    if (warp < 4) tc_fill_scales(tmem + ((uint32_t)(warp * 32) << 16));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == producer) {
        const bool one = tc_elect();
        int issued = 0, segs = 0;
        bool ok = true;
        TcItem it = first;
        for (int i = 0; i < nitem; i++, next(it)) {
            if (i == 0 || it.t == 0) {  // a new query pair: buffer segs & 1, free when segment segs - 2's MMAs are done
                const int a = segs & 1;
                if (segs >= 2) ok = mbar_wait_warp(&bar_a_free[a], ((segs >> 1) - 1) & 1);
                if (!ok) break;
                if (one) {
                    mbar_expect_tx(&bar_a[a], TC_QPAIR_BYTES);
                    bulk_g2s(sA + a * TC_QPAIR_BYTES, qa + (size_t)it.q * TC_QPAIR_BYTES, TC_QPAIR_BYTES, &bar_a[a]);
                }
                segs++;
            }
            const int s = i % TC_STAGES;
            if (i >= TC_STAGES) ok = mbar_wait_warp(&bar_empty[s], (i / TC_STAGES - 1) & 1);
            if (!ok) break;
            if (one) {
                mbar_expect_tx(&bar_full[s], TC_TTILE_BYTES);
                bulk_g2s(sB + s * TC_TTILE_BYTES, tb + (size_t)it.t * TC_TTILE_BYTES, TC_TTILE_BYTES, &bar_full[s]);
            }
            issued = i + 1;
        }
        // no copy may still be writing shared memory when the CTA ends:
        // wait (bounded) for the last phase issued on every barrier
        bool drained = true;
        for (int g = max(0, segs - 2); g < segs; g++) drained &= mbar_wait_warp(&bar_a[g & 1], (g >> 1) & 1);
        for (int i = max(0, issued - TC_STAGES); i < issued; i++)
            drained &= mbar_wait_warp(&bar_full[i % TC_STAGES], (i / TC_STAGES) & 1);
        if (one && !(ok && drained)) atomicOr(status, (ok ? 0 : 4) | (drained ? 0 : 32));
    } else if (warp >= issuer) {
        // issuer u takes every TC_ACCS-th of the items' query tiles (tile
        // j = 2 i + sub of item i where j % TC_ACCS == u) into accumulator u.  An MMA holds its warp until the tensor core takes it
        // and a wait on a barrier that is long complete still takes 85 cycles:
        // the waits of one warp pass beside the MMAs of the others.
        const int u = warp - issuer;
        const bool one = tc_elect();
        const uint32_t idesc = idesc_mxf4(TC_M, TC_N), d = tmem + (uint32_t)(u * TC_N);
        const uint64_t a0 = tc_operand(sA), b0 = tc_operand(sB);
        bool ok = true;
        int segs = 0, last = -1;  // last query tile issued
        TcItem it = first;
        for (int i = 0; i < nitem; i++) {
            if (i == 0 || it.t == 0) {  // every issuer follows every segment, with items in it or not
                ok = mbar_wait_warp(&bar_a[segs & 1], (segs >> 1) & 1);
                if (!ok) break;
                segs++;
            }
            const int s = i % TC_STAGES;
            for (int j = TC_QPAIR * i; j < TC_QPAIR * (i + 1); j++) {
                if (j % TC_ACCS != u) continue;
                const int ph = j / TC_ACCS;
                ok = mbar_wait_warp(&bar_full[s], (i / TC_STAGES) & 1);
                // the accumulator is free once the epilogue drained tile j - TC_ACCS
                if (ok && ph > 0) ok = mbar_wait_warp(&bar_acc_free[u], (ph - 1) & 1);
                if (!ok) break;
                tc_fence_after();
                const uint64_t ad = a0 + (uint32_t)((((segs - 1) & 1) * TC_QPAIR + (j & 1)) * (TC_QTILE_BYTES >> 4)),
                               bd = b0 + (uint32_t)(s * (TC_TTILE_BYTES >> 4));
                if (one) {
                    tc_tile_mma(d, ad, bd, idesc, tmem + TC_SCALE_COL);
                    tc_commit(&bar_empty[s]);  // the train buffer is free when both tiles' MMAs are done
                    tc_commit(&bar_acc[u]);    // and the accumulator ready
                }
                __syncwarp();
                last = j;
            }
            if (!ok) break;
            next(it);
            if (it.t == 0 && one) tc_commit(&bar_a_free[(segs - 1) & 1]);  // this issuer is done with the query pair
        }
        // TMEM is freed below: wait (bounded) until the last MMAs issued have
        // completed
        const bool drained = last < 0 || mbar_wait_warp(&bar_acc[u], (last / TC_ACCS) & 1);
        if (one && !(ok && drained)) atomicOr(status, (ok ? 0 : 8) | (drained ? 0 : 64));
    } else {
        // epilogue: warp w reads lanes 32 (w % 4).. of accumulator w / 4.  Keys
        // pack (distance << 23 | group index), so the lexicographic top-2 is
        // three min/max operations per group.  The dot products are exact
        // integers in [-256, 256]: adding 1.5 * 2^23 puts them in the low
        // mantissa bits, and 256 - dot = 2 * Hamming.
        const int quad = warp & 3, acc = warp >> 2;
        const int row = quad * 32 + lane;
        const uint32_t ta = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * TC_N);
        const int last_group = (nt - 1) / TC_GROUP;  // the groups after it hold no real row
        uint32_t k1[TC_QPAIR] = {0xFFFFFFFFu, 0xFFFFFFFFu}, k2[TC_QPAIR] = {0xFFFFFFFFu, 0xFFFFFFFFu};
        bool dead = false;
        TcItem it = first;
        for (int i = 0; i < nitem; i++) {
            const int q = it.q;
#pragma unroll
            for (int sub = 0; sub < TC_QPAIR; sub++) {
                const int j = TC_QPAIR * i + sub;
                if (j % TC_ACCS != acc || dead) continue;
                // one outcome for the warp: tcgen05.ld is a whole-warp
                // instruction (a warp that timed out reads nothing more, but
                // stays for the segments' barriers)
                if (!mbar_wait_warp(&bar_acc[acc], (j / TC_ACCS) & 1)) {
                    if (lane == 0) atomicOr(status, 16);
                    dead = true;
                } else {
                    tc_fence_after();
                    float m[TC_GROUPS];
                    // two groups at a time: the columns themselves land in
                    // registers that nothing reads
#pragma unroll
                    for (int g = 0; g < TC_GROUPS; g += 2) {
                        uint32_t r[2][TC_GROUP];
                        m[g] = tc_max32(ta + (uint32_t)(g * TC_GROUP), r[0]);
                        if (g + 1 < TC_GROUPS) m[g + 1] = tc_max32(ta + (uint32_t)((g + 1) * TC_GROUP), r[1]);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bar_acc_free[acc]);  // read: the next MMAs may overwrite it
                    const int g0 = it.t * TC_GROUPS;
#pragma unroll
                    for (int g = 0; g < TC_GROUPS; g++) {
                        const uint32_t twice = (uint32_t)(0x4B400000 + 256) - __float_as_uint(m[g] + 12582912.0f);
                        uint32_t key = (twice << 22) | (uint32_t)(g0 + g);
                        key = g0 + g <= last_group ? key : 0xFFFFFFFFu;
                        const uint32_t hi = max(k1[sub], key);
                        k1[sub] = min(k1[sub], key);
                        k2[sub] = min(k2[sub], hi);
                    }
                }
            }
            next(it);
            if (it.t == 0 || i + 1 == nitem) {
                // the segment's end: the accumulators' keys of every query row
#pragma unroll
                for (int sub = 0; sub < TC_QPAIR; sub++) {
                    s_part[acc][sub * TC_M + row] = make_uint2(k1[sub], k2[sub]);
                    k1[sub] = k2[sub] = 0xFFFFFFFFu;
                }
                asm volatile("bar.sync 1, %0;" ::"n"(32 * TC_EPI_WARPS) : "memory");
                if (threadIdx.x < TC_Q) {
                    const int qi = q * TC_Q + threadIdx.x;
                    uint2 b = s_part[0][threadIdx.x];
#pragma unroll
                    for (int p = 1; p < TC_ACCS; p++) {
                        const uint2 o = s_part[p][threadIdx.x];
                        const uint32_t hi = max(b.x, o.x);
                        b = make_uint2(min(b.x, o.x), min(min(b.y, o.y), hi));
                    }
                    const int slot = (int)((long)blockIdx.x - (long)q * tt / run);
                    if (qi < nq) partial[(size_t)slot * nq + qi] = b;
                }
                asm volatile("bar.sync 1, %0;" ::"n"(32 * TC_EPI_WARPS) : "memory");  // s_part is read
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == issuer) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// One warp per query: the two best groups over its pair's segments, then the
// two nearest of their rows, one row of each group per lane.
__global__ void __launch_bounds__(256) k_knn_tc_finish(const uint2* __restrict__ partial, const uint8_t* __restrict__ query,
                                                       const uint8_t* __restrict__ train, int nq, int nt, int tt, int run,
                                                       int* idx1, int* d1, int* idx2, int* d2) {
    const int qi = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (qi >= nq) return;
    const long q = qi / TC_Q;
    const int nslot = (int)(((q + 1) * tt - 1) / run - q * tt / run) + 1;
    uint32_t k1 = 0xFFFFFFFFu, k2 = 0xFFFFFFFFu;
    for (int s = lane; s < nslot; s += 32) {
        const uint2 o = partial[(size_t)s * nq + qi];
        const uint32_t hi = max(k1, o.x);
        k1 = min(k1, o.x);
        k2 = min(min(k2, o.y), hi);
    }
    const uint32_t g1 = __reduce_min_sync(0xffffffffu, k1);
    const uint32_t g2 = __reduce_min_sync(0xffffffffu, k1 == g1 ? k2 : k1);  // keys are distinct
    // 16-byte loads where both sets are aligned to them
    const bool wide = (((uintptr_t)query | (uintptr_t)train) & 15) == 0;
    auto load_row = [&](const uint8_t* p, uint4& lo, uint4& hi4) {
        if (wide) {
            lo = reinterpret_cast<const uint4*>(p)[0];
            hi4 = reinterpret_cast<const uint4*>(p)[1];
        } else {
            lo = make_uint4(load_u32(p), load_u32(p + 4), load_u32(p + 8), load_u32(p + 12));
            hi4 = make_uint4(load_u32(p + 16), load_u32(p + 20), load_u32(p + 24), load_u32(p + 28));
        }
    };
    uint4 a0, a1;
    load_row(query + 32 * (size_t)qi, a0, a1);
    auto row_key = [&](uint32_t g) -> uint32_t {
        const int j = (int)(g & 0x7FFFFFu) * TC_GROUP + lane;
        if (g == 0xFFFFFFFFu || j >= nt) return 0xFFFFFFFFu;
        uint4 t0, t1;
        load_row(train + 32 * (size_t)j, t0, t1);
        return ((uint32_t)hamming256(a0, a1, t0, t1) << 23) | (uint32_t)j;
    };
    uint32_t b1 = row_key(g1), b2 = row_key(g2);
    const uint32_t hi = max(b1, b2);
    b1 = min(b1, b2);
    b2 = hi;
    const uint32_t r1 = __reduce_min_sync(0xffffffffu, b1);
    const uint32_t r2 = __reduce_min_sync(0xffffffffu, b1 == r1 ? b2 : b1);
    if (lane == 0) {
        idx1[qi] = r1 == 0xFFFFFFFFu ? -1 : (int)(r1 & 0x7FFFFFu);
        d1[qi] = r1 == 0xFFFFFFFFu ? 0x7fffffff : (int)(r1 >> 23);
        idx2[qi] = r2 == 0xFFFFFFFFu ? -1 : (int)(r2 & 0x7FFFFFu);
        d2[qi] = r2 == 0xFFFFFFFFu ? 0x7fffffff : (int)(r2 >> 23);
    }
}

}  // namespace orbgpu

using namespace orbgpu;

// Tensor-core layout self-test: fills a query tile and a train tile with
// +-1 patterns of the given descriptors (host arrays, 128 and 256 rows) and
// returns the 128 x 256 dot products (host) and a status word.
extern "C" int orbgpu_debug_tc_probe(const uint8_t* q128, const uint8_t* t256, float* dots, int* status_out, int lbo,
                                     int sbo) {
    uint8_t *dq = nullptr, *dt = nullptr, *eq = nullptr, *et = nullptr;
    float* dd = nullptr;
    int* st = nullptr;
    ORBGPU_CUDA_TRY(cudaMalloc(&dq, 128 * 32));
    ORBGPU_CUDA_TRY(cudaMalloc(&dt, 256 * 32));
    ORBGPU_CUDA_TRY(cudaMalloc(&eq, TCP_QTILE_BYTES));
    ORBGPU_CUDA_TRY(cudaMalloc(&et, TCP_TTILE_BYTES));
    ORBGPU_CUDA_TRY(cudaMalloc(&dd, sizeof(float) * 128 * 256));
    ORBGPU_CUDA_TRY(cudaMalloc(&st, sizeof(int)));
    ORBGPU_CUDA_TRY(cudaMemcpy(dq, q128, 128 * 32, cudaMemcpyHostToDevice));
    ORBGPU_CUDA_TRY(cudaMemcpy(dt, t256, 256 * 32, cudaMemcpyHostToDevice));
    ORBGPU_CUDA_TRY(cudaMemset(st, 0, sizeof(int)));
    ORBGPU_CUDA_TRY(cudaMemset(dd, 0, sizeof(float) * 128 * 256));
    k_expand_fp8<<<128 * 16 / 256, 256>>>(dq, 128, TCP_M, eq);
    k_expand_fp8<<<256 * 16 / 256, 256>>>(dt, 256, TCP_N, et);
    const size_t smem = TCP_QTILE_BYTES + TCP_TTILE_BYTES;
    ORBGPU_CUDA_TRY(allow_max_dynamic_smem(k_tc_probe));
    k_tc_probe<<<1, 128, smem>>>(eq, et, dd, st, (uint32_t)lbo, (uint32_t)sbo);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    ORBGPU_CUDA_TRY(cudaDeviceSynchronize());
    ORBGPU_CUDA_TRY(cudaMemcpy(dots, dd, sizeof(float) * 128 * 256, cudaMemcpyDeviceToHost));
    ORBGPU_CUDA_TRY(cudaMemcpy(status_out, st, sizeof(int), cudaMemcpyDeviceToHost));
    cudaFree(dq);
    cudaFree(dt);
    cudaFree(eq);
    cudaFree(et);
    cudaFree(dd);
    cudaFree(st);
    return ORBGPU_OK;
}

// The kNN kernel's tile product: nq <= 128 queries against nt <= 160 train rows
// (host arrays), expanded as for a search; the last row of a set repeats in its
// tile.
extern "C" int orbgpu_debug_knn_tile(const uint8_t* query, int nq, const uint8_t* train, int nt, float* dots,
                                     float* maxima, int* status_out) {
    if (!query || !train || nq < 1 || nq > TC_M || nt < 1 || nt > TC_N || !dots || !maxima || !status_out)
        return ORBGPU_ERR_BAD_ARG;
    uint8_t *dq = nullptr, *dt = nullptr, *operands = nullptr;
    float* out = nullptr;
    int* st = nullptr;
    const size_t nd = (size_t)TC_M * TC_N, nm = (size_t)TC_M * TC_GROUPS;
    ORBGPU_CUDA_TRY(cudaMalloc(&dq, 32 * (size_t)nq));
    ORBGPU_CUDA_TRY(cudaMalloc(&dt, 32 * (size_t)nt));
    ORBGPU_CUDA_TRY(cudaMalloc(&operands, TC_QTILE_BYTES + TC_TTILE_BYTES));
    ORBGPU_CUDA_TRY(cudaMalloc(&out, sizeof(float) * (nd + nm)));
    ORBGPU_CUDA_TRY(cudaMalloc(&st, sizeof(int)));
    ORBGPU_CUDA_TRY(cudaMemcpy(dq, query, 32 * (size_t)nq, cudaMemcpyHostToDevice));
    ORBGPU_CUDA_TRY(cudaMemcpy(dt, train, 32 * (size_t)nt, cudaMemcpyHostToDevice));
    ORBGPU_CUDA_TRY(cudaMemset(out, 0, sizeof(float) * (nd + nm)));
    const long qth = TC_QTILE_BYTES / 16, tth = TC_TTILE_BYTES / 16;
    k_expand_fp4<<<(unsigned)((qth + tth + 255) / 256), 256>>>(dq, nq, qth, operands, dt, nt, tth,
                                                             operands + TC_QTILE_BYTES, st);
    ORBGPU_CUDA_TRY(allow_max_dynamic_smem(k_knn_tile_probe));
    k_knn_tile_probe<<<1, 128, TC_QTILE_BYTES + TC_TTILE_BYTES>>>(operands, operands + TC_QTILE_BYTES, out, out + nd, st);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    ORBGPU_CUDA_TRY(cudaDeviceSynchronize());
    ORBGPU_CUDA_TRY(cudaMemcpy(dots, out, sizeof(float) * nd, cudaMemcpyDeviceToHost));
    ORBGPU_CUDA_TRY(cudaMemcpy(maxima, out + nd, sizeof(float) * nm, cudaMemcpyDeviceToHost));
    ORBGPU_CUDA_TRY(cudaMemcpy(status_out, st, sizeof(int), cudaMemcpyDeviceToHost));
    cudaFree(dq);
    cudaFree(dt);
    cudaFree(operands);
    cudaFree(out);
    cudaFree(st);
    return ORBGPU_OK;
}

// The tensor-core kNN (algo 1 of orbgpu_knn2); see orbgpu.h.
int orbgpu_knn2_tc(orbgpu_matcher* m, const uint8_t* query, int nq, const uint8_t* train, int nt, int* idx1, int* d1,
                   int* idx2, int* d2) {
    if (nq <= 0 || nt <= 0) return ORBGPU_ERR_BAD_ARG;  // the caller answers empty sets
    cudaStream_t st = orbgpu_matcher_stream_internal(m);
    const int nsm = nsm_of_current_device();
    const int pairs = (nq + TC_Q - 1) / TC_Q, tt = (nt + TC_N - 1) / TC_N;
    const long items = (long)pairs * tt;
    const int run = (int)((items + nsm - 1) / nsm);
    const int ctas = (int)((items + run - 1) / run);
    const int slots = (tt + run - 1) / run + 1;  // segments of one query pair, at most
    const size_t q_bytes = (size_t)pairs * TC_QPAIR_BYTES, t_bytes = (size_t)tt * TC_TTILE_BYTES,
                 p_bytes = (sizeof(uint2) * (size_t)nq * slots + 255) & ~(size_t)255;
    KnnWorkspace work(m);
    const int rc = work.take(q_bytes + t_bytes + p_bytes + 256);
    if (rc != ORBGPU_OK) return rc;
    uint8_t* eq = work.data();
    uint8_t* et = eq + q_bytes;
    uint2* partial = (uint2*)(et + t_bytes);
    int* status = (int*)(et + t_bytes + p_bytes);
    const long qth = (long)(q_bytes / 16), tth = (long)(t_bytes / 16);
    k_expand_fp4<<<(unsigned)((qth + tth + 255) / 256), 256, 0, st>>>(query, nq, qth, eq, train, nt, tth, et, status);
    const size_t smem = 2 * TC_QPAIR_BYTES + TC_STAGES * TC_TTILE_BYTES;
    ORBGPU_CUDA_TRY(allow_max_dynamic_smem(k_knn_tc));
    k_knn_tc<<<ctas, TC_THREADS, smem, st>>>(eq, et, nq, nt, items, tt, run, partial, status);
    k_knn_tc_finish<<<(nq + 7) / 8, 256, 0, st>>>(partial, query, train, nq, nt, tt, run, idx1, d1, idx2, d2);
    ORBGPU_CUDA_TRY(cudaGetLastError());
    ORBGPU_CUDA_TRY(cudaMemcpyAsync(work.pinned(), status, sizeof(int), cudaMemcpyDeviceToHost, st));
    ORBGPU_CUDA_TRY(cudaStreamSynchronize(st));
    const int hstatus = work.pinned()[0];
    if (hstatus) {
        char msg[96];
        std::snprintf(msg, sizeof(msg), "tensor-core kNN wait timed out (status 0x%x)", hstatus);
        orbgpu_set_last_error(msg, __FILE__, __LINE__);
        return ORBGPU_ERR_TIMEOUT;
    }
    return ORBGPU_OK;
}
