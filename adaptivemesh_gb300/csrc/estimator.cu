// estimator.cu -- the learned refinement / error estimator: a small 3-D convolutional network run per
// tile (one domain), trained on the GPU by the kernels below.  No counterpart in the reference,
// whose refinement criterion is a per-octant gradient and curvature threshold
// (SimpleWave.h:91-187, 228-248); here that plain criterion stays both the fallback and the judge
// of the network's decisions (evolve_sim.cu, amr_sim_regrid).
//
// Network (per tile, input 3 x 8^3 features):
//   conv1  3 -> 16 channels, 3x3x3, padding 1, stride 1, ReLU      -> 16 x 8^3
//   conv2  16 -> 16 channels, 3x3x3, padding 1, stride 2, ReLU     -> 16 x 4^3 = 1024
//   fc1    1024 -> 32, ReLU
//   fc2    32 -> 1 (the predicted log10 truncation error of the tile)
// The convolutions and the weight gradients run as GEMMs on the fifth-generation tensor cores
// (tcgen05.mma kind::f16, BF16 operands in shared memory, FP32 accumulation in Tensor Memory) whose
// operands are gathered from the activations.
// Master weights, gradients and the Adam moments are FP32; the products' operands (weights,
// activations, back-propagated gradients) are rounded to BF16.
//
// Layouts: activations are position-major, channel-last ([tile][position][channel]); receptive-field
// index j = channel * 27 + (dz * 9 + dy * 3 + dx) for the tap at offset (dx, dy, dz) - 1; conv1's 81
// are padded to 96 with zeros.  The flat parameter vector is W1[96][16], b1[16],
// W2[432][16], b2[16], W3[1024][32], b3[32], W4[32], b4[1] (row-major, K rows by N columns).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "amr_device.cuh"
#include "capi_internal.h"
#include "kernels.h"
#include "tcgen05.cuh"

namespace amr {

namespace {

using bf16 = __nv_bfloat16;

constexpr int kIn = 3, kC1 = 16, kC2 = 16, kF = 32;
constexpr int kP1 = 512, kP2 = 64;                 // positions after conv1 (8^3) and conv2 (4^3)
constexpr int kK1 = 96, kK1Real = kIn * 27, kK2 = kC1 * 27, kK3 = kP2 * kC2;   // 96, 432, 1024
constexpr size_t kOffW1 = 0, kOffB1 = kOffW1 + kK1 * kC1, kOffW2 = kOffB1 + kC1, kOffB2 = kOffW2 + kK2 * kC2,
                 kOffW3 = kOffB2 + kC2, kOffB3 = kOffW3 + (size_t)kK3 * kF, kOffW4 = kOffB3 + kF,
                 kOffB4 = kOffW4 + kF, kParams = kOffB4 + 1;

// ------------------------------------------------------------------ BF16 GEMM on the tensor cores
// C = A B for one 128 x NT tile (NT = 16 or 32) and one range of K per CTA of 4 warps, on the
// fifth-generation tensor cores: per K block of 64 the threads stage A (128 x 64) and B (NT x 64) into
// shared memory as K-major core matrices, one thread issues four tcgen05.mma of K = 16 into a TMEM
// accumulator and commits them to an mbarrier, and after the last block each warp reads its 32 rows of
// the accumulator back with tcgen05.ld and hands each row to the epilogue.  Every wait is bounded; a
// wait that runs out raises *err, waits once more for the MMAs in flight and frees the TMEM.
//
// The operands are functors: thread t stages row t of A, eight K values (16 bytes) at a time, so that
// the convolutions gather their receptive fields straight from the activations (no im2col matrix in
// memory, 98 KB a tile for conv1 before) and a row's geometry is computed once.  G blocks are staged at a
// time, all their loads in flight together, and the next G are loaded while they are multiplied: a block's
// load latency, paid 16 times, was most of fc1's time (one or two CTAs; 36 us for 256 tiles, 22 with four).  A
// convolution's K is a template parameter and its loop unrolled, so that channel, tap and offset of every
// gathered value are constants (conv2 21.6 -> 17.7 us, conv1 18.2 -> 9.5, 256 tiles).  The epilogue takes the
// bias, the ReLU and its backward form, which were passes of their own.
constexpr int kGemmM = 128, kGemmK = 64;

struct __align__(16) Chunk {   // eight consecutive K values of one row
    bf16 v[8];
};
__device__ __forceinline__ Chunk zero_chunk() {
    Chunk c;
    *reinterpret_cast<uint4*>(&c) = make_uint4(0u, 0u, 0u, 0u);
    return c;
}

template <int NT, int KC, int G, class A, class B, class Epilogue>
__global__ void __launch_bounds__(128) k_gemm_bf16(const A fa, const B fb, const Epilogue epi, int k_runtime, int* err) {
    grid_dependency();
    static_assert(NT == 16 || NT == 32, "M = 128 tiles take N in multiples of 16; 32 TMEM columns");
    constexpr int MT = kGemmM, KT = kGemmK, BC = NT * KT / 8 / 128;   // chunks of B per thread and block
    constexpr uint32_t LBO = 128u, SBO = (KT / 8) * 128u;   // bytes between core matrices along K / M
    extern __shared__ __align__(1024) unsigned char smem_raw[];   // G blocks of A, then of B
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = tid / 32;
    const int m = blockIdx.x * MT + tid, n0 = blockIdx.y * NT;
    if (warp == 0) tmem_alloc(&s_tmem, 32u);   // the 128 x NT FP32 accumulator
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
        s_fail = 0;
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 0) tmem_relinquish();
    const uint32_t tmem = s_tmem;
    constexpr uint32_t idesc = umma_idesc_bf16_f32(MT, NT);
    // chunk k of row r: core matrix (r / 8, k) of eight 16-byte rows, row r % 8
    auto at = [](int r, int k) { return (r >> 3) * (KT / 8) * 8 + k * 8 + (r & 7); };
    Chunk* const a16 = reinterpret_cast<Chunk*>(smem_raw);
    Chunk* const b16 = a16 + G * MT * KT / 8;
    uint32_t phase = 0;
    const int nkb = ((KC ? KC : k_runtime) + KT - 1) / KT;
    // Thread t stages row t where a row's geometry costs; where its K values are contiguous, a warp takes eight
    // rows and four chunks of each, 64 bytes of a line instead of 16 (and no two rows' banks meet).
    const auto row = fa.row(A::kByRow ? 0 : m);
    auto row_of = [&](int i) { return A::kByRow ? 8 * ((warp * (KT / 8) + i) / 2) + (tid & 7) : tid; };
    auto chunk_of = [&](int i) { return A::kByRow ? 4 * (i & 1) + (tid % 32) / 8 : i; };
    Chunk ca[G][KT / 8], cb[G][BC];
    auto load = [&](int kb) {   // blocks kb .. kb + G - 1, as far as there are
#pragma unroll
        for (int j = 0; j < G; j++) {
            if (kb + j >= nkb) break;
            const int k0 = (kb + j) * KT;
#pragma unroll
            for (int i = 0; i < KT / 8; i++) {
                if constexpr (A::kByRow) ca[j][i] = fa(blockIdx.x * MT + row_of(i), k0 + 8 * chunk_of(i));
                else ca[j][i] = fa(row, k0 + 8 * i);
            }
#pragma unroll
            for (int i = 0; i < BC; i++) {
                const int e = tid + 128 * i;
                cb[j][i] = fb(n0 + e % NT, k0 + 8 * (e / NT));
            }
        }
    };
    auto group = [&](int kb) {
#pragma unroll
        for (int j = 0; j < G; j++) {
            if (kb + j >= nkb) break;
#pragma unroll
            for (int i = 0; i < KT / 8; i++) a16[j * MT * KT / 8 + at(row_of(i), chunk_of(i))] = ca[j][i];
#pragma unroll
            for (int i = 0; i < BC; i++) b16[j * NT * KT / 8 + at((tid + 128 * i) % NT, (tid + 128 * i) / NT)] = cb[j][i];
        }
        fence_proxy_async_smem();   // these writes, visible to the tensor core
        __syncthreads();
        if (tid == 0) {
            tc_fence_after_sync();
            const uint32_t a0 = smem_addr(a16), b0 = smem_addr(b16);
#pragma unroll
            for (int j = 0; j < G; j++) {
                if (kb + j >= nkb) break;
#pragma unroll
                for (int kk = 0; kk < KT / 16; kk++)   // K = 16 per MMA: two core matrices along K
                    umma_bf16(tmem, umma_desc_kmajor(a0 + j * MT * KT * 2 + kk * 2 * LBO, LBO, SBO),
                              umma_desc_kmajor(b0 + j * NT * KT * 2 + kk * 2 * LBO, LBO, SBO), idesc, kb > 0 || j > 0 || kk > 0);
            }
            umma_commit(&bar);
        }
        load(kb + G);
        // the group's MMAs have read its operands once the barrier's phase completes
        const bool ok = mbar_wait(&bar, phase);
        phase ^= 1u;
        if (!ok) s_fail = 1;
        __syncthreads();
        return s_fail == 0;
    };
    load(0);
    if constexpr (KC != 0 && KC <= 8 * KT) {
#pragma unroll
        for (int kb = 0; kb < nkb; kb += G)
            if (!group(kb)) break;
    } else {
#pragma unroll 1
        for (int kb = 0; kb < nkb; kb += G)
            if (!group(kb)) break;
    }
    if (!s_fail) {
        tc_fence_after_sync();
        float v[NT];
        const uint32_t row_addr = tmem + ((uint32_t)(warp * 32) << 16);   // lanes 32 w .. 32 w + 31
        tmem_ld16(row_addr, v);
        if constexpr (NT == 32) tmem_ld16(row_addr + 16u, v + 16);
        epi(m, n0, v);
    } else if (tid == 0) {
        atomicExch(err, 1);
        mbar_wait(&bar, phase ^ 1u);   // the MMAs of the group whose wait gave up
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, 32u);
    }
}

// C (rows x cols) over all of K; KC: K where it is known, G: K blocks staged at a time
template <int NT, int KC, int G, class A, class B, class Epilogue>
cudaError_t gemm(const A& fa, const B& fb, const Epilogue& epi, int rows, int cols, int K, cudaStream_t st) {
    if (rows <= 0 || K <= 0) return cudaSuccess;
    int* err = device_error_flag();
    if (!err) return cudaErrorMemoryAllocation;
    constexpr size_t smem = (size_t)G * (kGemmM + NT) * kGemmK * sizeof(bf16);
    static std::atomic<uint64_t> configured{0};
    const cudaError_t e = ensure_smem_limit(k_gemm_bf16<NT, KC, G, A, B, Epilogue>, smem, configured);
    if (e != cudaSuccess) return e;
    return launch_dependent(true, k_gemm_bf16<NT, KC, G, A, B, Epilogue>,
                            dim3((unsigned)((rows + kGemmM - 1) / kGemmM), (unsigned)((cols + NT - 1) / NT)), 128, smem, st, fa, fb,
                            epi, K, err);
}

// ------------------------------------------------------------------ weight gradients of the convolutions
// dW = A^T dY contracts over every position of the batch (K = 32 768 for conv1 with 64 tiles) into 96 or 432
// rows of 16.  One CTA per 128 rows staged and multiplied all of K block after block: 2 529 us for
// conv1's.  The sums stay in that one order (K ascending, 16 at a time), so that a training run's
// losses do not change; instead k_pack lays both operands out in parallel, as the core matrices the
// tensor core reads, and k_stream_gemm, one CTA per 8 rows, streams its slabs through a ring of bulk
// copies with nothing between the MMAs.  The chain of dependent MMAs is what is left: 2 048 of them for
// conv1's 64 tiles, 50 ns each, 102 us, whatever few of a 128 x 16 x 16 MMA's rows are used (ranges of K
// summed afterwards took 12 us and changed the last bits of the gradients).
//
// One Adam step of 64 tiles, GB300: 2 730 -> 215 us, 27 -> 13 launches, every bit as before; forward
// pass of 256 tiles 330 -> 52 us.
constexpr int kSlabRows = 8;
constexpr int kSlabA = kSlabRows * kGemmK * 2, kSlabB = 16 * kGemmK * 2;   // bytes per K block

// A^T's slabs [row / 8][K block][k chunk][row % 8] and dY's [K block][n / 8][k chunk][n % 8], chunks of
// eight K values; `rows` a multiple of 8, K a multiple of 64.
template <class A, class B>
__device__ __forceinline__ void pack_chunk(const A& fa, const B& fb, int rows, int K, int i, Chunk* pa, Chunk* pb) {
    const int nkb = K / kGemmK, na = rows * nkb * 8;
    if (i < na) {
        const int r = i % 8, kc = (i / 8) % 8, kb = (i / 64) % nkb, g = i / 64 / nkb;
        pa[i] = fa(fa.row(8 * g + r), kb * kGemmK + 8 * kc);
    } else if (i < na + 16 * nkb * 8) {
        const int e = i - na, r = e % 8, kc = (e / 8) % 8, g = (e / 64) % 2, kb = e / 128;
        pb[e] = fb(8 * g + r, kb * kGemmK + 8 * kc);
    }
}
template <class A1, class B1, class A2, class B2>
__global__ void __launch_bounds__(256) k_pack(const A1 a1, const B1 b1, int rows1, int K1, Chunk* pa1, Chunk* pb1, const A2 a2,
                                              const B2 b2, int rows2, int K2, Chunk* pa2, Chunk* pb2) {
    grid_dependency();
    const int n1 = (rows1 + 16) * (K1 / kGemmK) * 8, i = blockIdx.x * 256 + threadIdx.x;
    if (i < n1) pack_chunk(a1, b1, rows1, K1, i, pa1, pb1);
    else pack_chunk(a2, b2, rows2, K2, i - n1, pa2, pb2);
}
struct StreamGemm {
    const Chunk* a;
    const Chunk* b;
    float* out;   // [rows][16]
    int rows, nkb;
};
// K blocks per ring stage, stages; the MMAs' rows past a slab's 8 read what lies behind it in shared
// memory (their results are not used): 16 KB more than the ring.
constexpr int kStageBlocks = 4, kStages = 6;
constexpr size_t kStreamSmem = (size_t)kStages * kStageBlocks * (kSlabA + kSlabB) + 16384u;
__global__ void __launch_bounds__(64) k_stream_gemm(const StreamGemm g1, const StreamGemm g2, int* err) {
    grid_dependency();
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages], done;
    __shared__ uint32_t s_tmem;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const bool first = (int)blockIdx.x < g1.rows / kSlabRows;
    const StreamGemm& g = first ? g1 : g2;
    const int slab = first ? (int)blockIdx.x : (int)blockIdx.x - g1.rows / kSlabRows;
    if (warp == 0) tmem_alloc(&s_tmem, 32u);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(&done, 1);
        mbar_fence_init();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 0) tmem_relinquish();
    const uint32_t tmem = s_tmem;
    constexpr uint32_t idesc = umma_idesc_bf16_f32(kGemmM, 16), LBO = 128u, SBO = (kGemmK / 8) * 128u;
    constexpr int kStageA = kStageBlocks * kSlabA;
    const int ns = (g.nkb + kStageBlocks - 1) / kStageBlocks;
    bool ok = true;
    if (warp == 0 && lane == 0) {   // producer
        for (int i = 0; i < ns && ok; i++) {
            const int s = i % kStages, n = min(kStageBlocks, g.nkb - i * kStageBlocks);
            if (i >= kStages) ok = mbar_wait(&empty[s], (uint32_t)(i / kStages - 1) & 1u);
            if (!ok) break;
            unsigned char* dst = smem + (size_t)s * kStageBlocks * (kSlabA + kSlabB);
            mbar_arrive_expect_tx(&full[s], (uint32_t)(n * (kSlabA + kSlabB)));
            bulk_g2s(dst, g.a + ((size_t)slab * g.nkb + (size_t)i * kStageBlocks) * (kSlabA / 16), (uint32_t)(n * kSlabA), &full[s]);
            bulk_g2s(dst + kStageA, g.b + (size_t)i * kStageBlocks * (kSlabB / 16), (uint32_t)(n * kSlabB), &full[s]);
        }
    } else if (warp == 1 && lane == 0) {   // the MMAs, in the order of K
        for (int i = 0; i < ns && ok; i++) {
            const int s = i % kStages, n = min(kStageBlocks, g.nkb - i * kStageBlocks);
            ok = mbar_wait(&full[s], (uint32_t)(i / kStages) & 1u);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t a0 = smem_addr(smem + (size_t)s * kStageBlocks * (kSlabA + kSlabB)), b0 = a0 + kStageA;
            for (int k = 0; k < n; k++)
#pragma unroll
                for (int kk = 0; kk < kGemmK / 16; kk++)
                    umma_bf16(tmem, umma_desc_kmajor(a0 + k * kSlabA + kk * 2 * LBO, LBO, SBO),
                              umma_desc_kmajor(b0 + k * kSlabB + kk * 2 * LBO, LBO, SBO), idesc, i > 0 || k > 0 || kk > 0);
            umma_commit(&empty[s]);
        }
        umma_commit(&done);   // also after a wait gave up: the MMAs in flight
    }
    __syncwarp();
    const bool fin = mbar_wait(&done, 0u) && ok;
    // every copy issued lands before the CTA leaves: in a normal run the MMAs consumed them all
    const bool good = __syncthreads_and(fin);
    if (!good) {
        if (threadIdx.x == 0) {
            atomicExch(err, 1);
            for (int s = 0; s < kStages; s++)   // both parities: one of them is the stage's last request (bounded waits)
                for (uint32_t q = 0; q < 2; q++) mbar_wait(&full[s], q, 4096u);
        }
        __syncthreads();
    } else if (warp == 0) {
        tc_fence_after_sync();
        float v[16];
        tmem_ld16(tmem, v);   // lanes 0 .. 31: the slab's rows are the first 8
        if (lane < kSlabRows) {
            float4* o = reinterpret_cast<float4*>(g.out + (size_t)(slab * kSlabRows + lane) * 16);
#pragma unroll
            for (int n = 0; n < 4; n++) o[n] = make_float4(v[4 * n], v[4 * n + 1], v[4 * n + 2], v[4 * n + 3]);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, 32u);
    }
}

// ------------------------------------------------------------------ the GEMMs' operands
// conv1's receptive fields: row = (tile, position), K = channel * 27 + tap, from the features
struct Conv1A {
    static constexpr bool kByRow = false;
    const float* x;
    int rows;
    struct Row { const float* p; uint32_t taps; };   // the position's cell in channel 0, the taps inside the tile
    __device__ Row row(int m) const {
        Row r{x, 0u};
        if (m >= rows) return r;
        const int pos = m % kP1, px = pos % 8, py = (pos / 8) % 8, pz = pos / 64;
        r.p = x + (int64_t)(m / kP1) * kIn * kP1 + pos;
#pragma unroll
        for (int t = 0; t < 27; t++) {
            const int x0 = px + t % 3 - 1, y0 = py + (t / 3) % 3 - 1, z0 = pz + t / 9 - 1;
            if (x0 >= 0 && x0 < 8 && y0 >= 0 && y0 < 8 && z0 >= 0 && z0 < 8) r.taps |= 1u << t;
        }
        return r;
    }
    __device__ Chunk operator()(const Row& r, int k) const {
        Chunk c;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int j = k + i, ch = j / 27, t = j - 27 * ch;
            float v = 0.f;
            if (j < kK1Real && (r.taps >> t & 1u)) v = r.p[ch * kP1 + (t % 3 - 1) + ((t / 3) % 3 - 1) * 8 + (t / 9 - 1) * 64];
            c.v[i] = __float2bfloat16_rn(v);
        }
        return c;
    }
};
// A weight matrix [K][cols] as the B operand: row n of its transpose
template <int COLS, int KREAL>
struct WeightB {
    const bf16* w;
    __device__ Chunk operator()(int n, int k) const {
        Chunk c;
#pragma unroll
        for (int i = 0; i < 8; i++)   // (whole blocks of K need no test, which would part the loads)
            c.v[i] = KREAL % kGemmK == 0 || k + i < KREAL ? w[(k + i) * COLS + n] : __float2bfloat16_rn(0.f);
        return c;
    }
};
struct Conv2A {
    static constexpr bool kByRow = false;
    const bf16* h1;   // [tile][512][16]
    int rows;
    struct Row { const bf16* p; uint32_t taps; };
    __device__ Row row(int m) const {
        Row r{h1, 0u};
        if (m >= rows) return r;
        const int o = m % kP2, px = 2 * (o % 4), py = 2 * ((o / 4) % 4), pz = 2 * (o / 16);   // stride 2
        r.p = h1 + ((int64_t)(m / kP2) * kP1 + (pz * 8 + py) * 8 + px) * kC1;
#pragma unroll
        for (int t = 0; t < 27; t++) {
            const int x0 = px + t % 3 - 1, y0 = py + (t / 3) % 3 - 1, z0 = pz + t / 9 - 1;
            if (x0 >= 0 && x0 < 8 && y0 >= 0 && y0 < 8 && z0 >= 0 && z0 < 8) r.taps |= 1u << t;
        }
        return r;
    }
    __device__ Chunk operator()(const Row& r, int k) const {
        Chunk c;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int j = k + i, ch = j / 27, t = j - 27 * ch;
            c.v[i] = j < kK2 && (r.taps >> t & 1u) ? r.p[((t % 3 - 1) + ((t / 3) % 3 - 1) * 8 + (t / 9 - 1) * 64) * kC1 + ch]
                                                   : __float2bfloat16_rn(0.f);
        }
        return c;
    }
};
// Rows of a matrix whose K = KREAL values are contiguous: [row][KREAL]
template <int KREAL>
struct RowsA {
    static constexpr bool kByRow = true;
    const bf16* p;
    int rows;
    struct Row { const bf16* p; bool ok; };
    __device__ Row row(int m) const { return Row{p + (int64_t)(m < rows ? m : 0) * KREAL, m < rows}; }
    __device__ Chunk operator()(const Row& r, int k) const {   // loaded in any case: a branch would part the loads
        const uint4 c = *reinterpret_cast<const uint4*>(r.p + (KREAL % kGemmK == 0 || k < KREAL ? k : 0));
        const bool ok = r.ok && (KREAL % kGemmK == 0 || k < KREAL);
        Chunk z;
        *reinterpret_cast<uint4*>(&z) = make_uint4(ok ? c.x : 0u, ok ? c.y : 0u, ok ? c.z : 0u, ok ? c.w : 0u);
        return z;
    }
    __device__ Chunk operator()(int n, int k) const { return (*this)(row(n), k); }   // row n: of A by rows, or of B
};
// The transposed receptive fields for the weight gradients: row = K index of the forward pass,
// K = (tile, position)
struct Conv1At {
    const float* x;
    struct Row { int ch, dx, dy, dz; };   // ch = -1: a padding row
    __device__ Row row(int j) const {
        const int t = j % 27;
        return Row{j < kK1Real ? j / 27 : -1, t % 3 - 1, (t / 3) % 3 - 1, t / 9 - 1};
    }
    __device__ Chunk operator()(const Row& r, int k) const {   // eight positions: one row of x
        const int pos = k % kP1, y = (pos / 8) % 8 + r.dy, z = pos / 64 + r.dz;
        if (r.ch < 0 || y < 0 || y >= 8 || z < 0 || z >= 8) return zero_chunk();
        const float* p = x + ((int64_t)(k / kP1) * kIn + r.ch) * kP1 + (z * 8 + y) * 8 + r.dx;
        Chunk c;
#pragma unroll
        for (int i = 0; i < 8; i++) c.v[i] = __float2bfloat16_rn(i + r.dx >= 0 && i + r.dx < 8 ? p[i] : 0.f);
        return c;
    }
};
struct Conv2At {
    const bf16* h1;
    struct Row { int ch, dx, dy, dz; };
    __device__ Row row(int j) const {
        const int t = j % 27;
        return Row{j < kK2 ? j / 27 : -1, t % 3 - 1, (t / 3) % 3 - 1, t / 9 - 1};
    }
    __device__ Chunk operator()(const Row& r, int k) const {   // eight outputs: two rows of four
        const int o = k % kP2, z = 2 * (o / 16) + r.dz;
        if (r.ch < 0 || z < 0 || z >= 8) return zero_chunk();
        const bf16* p = h1 + ((int64_t)(k / kP2) * kP1 + z * 64) * kC1 + r.ch;
        Chunk c;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int x = 2 * (i % 4) + r.dx, y = 2 * ((o / 4) % 4 + i / 4) + r.dy;
            c.v[i] = x >= 0 && x < 8 && y >= 0 && y < 8 ? p[(y * 8 + x) * kC1] : __float2bfloat16_rn(0.f);
        }
        return c;
    }
};
// Rows of a [K][cols] matrix read down its columns (H2 and the back-propagated gradients)
template <int COLS>
struct ColumnsT {
    static constexpr bool kByRow = false;
    const bf16* p;
    int K;
    struct Row { const bf16* p; };
    __device__ Row row(int m) const { return Row{p + (m < COLS ? m : 0)}; }
    __device__ Chunk operator()(const Row& r, int k) const {
        Chunk c;
#pragma unroll
        for (int i = 0; i < 8; i++) c.v[i] = k + i < K ? r.p[(int64_t)(k + i) * COLS] : __float2bfloat16_rn(0.f);
        return c;
    }
    __device__ Chunk operator()(int n, int k) const { return (*this)(row(n), k); }
};

// ------------------------------------------------------------------ the GEMMs' epilogues
// z = y + bias (kept for the backward pass where z is set), h = bf16(relu(z)); NT columns
template <int NT>
struct BiasRelu {
    const float* bias;
    float* z;
    bf16* h;
    int rows;
    __device__ void operator()(int m, int, float* v) const {
        if (m >= rows) return;
#pragma unroll
        for (int n = 0; n < NT; n += 8) {
            Chunk c;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                v[n + i] = v[n + i] + bias[n + i];
                c.v[i] = __float2bfloat16_rn(fmaxf(v[n + i], 0.f));
            }
            *reinterpret_cast<Chunk*>(h + (int64_t)m * NT + n) = c;
        }
        if (z)
#pragma unroll
            for (int n = 0; n < NT; n += 4)
                *reinterpret_cast<float4*>(z + (int64_t)m * NT + n) = make_float4(v[n], v[n + 1], v[n + 2], v[n + 3]);
    }
};
// the tile of a rows x COLS matrix
template <int NT, int COLS>
struct Store {
    float* out;
    int rows;
    __device__ void operator()(int m, int n0, const float* v) const {
        if (m >= rows) return;
#pragma unroll
        for (int n = 0; n < NT; n += 4)
            if (n0 + n < COLS)
                *reinterpret_cast<float4*>(out + (int64_t)m * COLS + n0 + n) = make_float4(v[n], v[n + 1], v[n + 2], v[n + 3]);
    }
};
// gradient through the ReLU: dz = dh * (z > 0), FP32 (for the bias gradient) and BF16 (an operand)
template <int NT, int COLS>
struct ReluBack {
    const float* z;
    float* dz;
    bf16* dzb;
    int rows;
    __device__ void operator()(int m, int n0, float* v) const {
        if (m >= rows) return;
        const int64_t o = (int64_t)m * COLS + n0;
#pragma unroll
        for (int n = 0; n < NT; n += 8) {
            Chunk c;
#pragma unroll
            for (int i = 0; i < 8; i += 4) {
                const float4 zz = *reinterpret_cast<const float4*>(z + o + n + i);
                const float zv[4] = {zz.x, zz.y, zz.z, zz.w};
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    v[n + i + q] = zv[q] > 0.f ? v[n + i + q] : 0.f;
                    c.v[i + q] = __float2bfloat16_rn(v[n + i + q]);
                }
                *reinterpret_cast<float4*>(dz + o + n + i) = make_float4(v[n + i], v[n + i + 1], v[n + i + 2], v[n + i + 3]);
            }
            *reinterpret_cast<Chunk*>(dzb + o + n) = c;
        }
    }
};

// ------------------------------------------------------------------ the last layer, sums and Adam
// fc2 and the loss, a warp per tile: out[b] = h3[b] . w4 + b4 (in the order of k); with targets, dout = 2 (out - t) / B,
// the loss terms, and dZ3 = (dout w4) through fc1's ReLU (FP32 and BF16)
__global__ void __launch_bounds__(128) k_fc2(const bf16* __restrict__ h3, const float* __restrict__ w4, const float* __restrict__ b4,
                                             int B, float* __restrict__ out, const float* __restrict__ target,
                                             float* __restrict__ dout, float* __restrict__ sq, const float* __restrict__ z3,
                                             float* __restrict__ dz3, bf16* __restrict__ dz3b) {
    grid_dependency();
    const int b = blockIdx.x * 4 + threadIdx.x / 32, k = threadIdx.x % 32;
    if (b >= B) return;
    const float h = __bfloat162float(h3[(int64_t)b * kF + k]), w = __bfloat162float(__float2bfloat16_rn(w4[k]));
    float s = b4[0];
#pragma unroll
    for (int i = 0; i < kF; i++) s = fmaf(__shfl_sync(0xffffffffu, h, i), __shfl_sync(0xffffffffu, w, i), s);
    if (k == 0) out[b] = s;
    if (!target) return;
    const float d = s - target[b], g = 2.f * d / (float)B;
    if (k == 0) {
        dout[b] = g;
        sq[b] = d * d;
    }
    const int64_t i = (int64_t)b * kF + k;
    const float v = z3[i] > 0.f ? g * w : 0.f;
    dz3[i] = v;
    dz3b[i] = __float2bfloat16_rn(v);
}
// conv2's col2im through conv1's ReLU: dH1[tile][pos][c] = sum of dA2 over the (output, tap) pairs reading
// it, gathered in a fixed order (no atomics); dZ1 in FP32 and BF16
__global__ void __launch_bounds__(256) k_col2im2(const float* __restrict__ da, const float* __restrict__ z1, int B,
                                                 float* __restrict__ dz1, bf16* __restrict__ dz1b) {
    grid_dependency();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)B * kP1 * kC1) return;
    const int c = (int)(i % kC1);
    const int64_t row = i / kC1;
    const int b = (int)(row / kP1), pos = (int)(row % kP1);
    const int px = pos % 8, py = (pos / 8) % 8, pz = pos / 64;
    float s = 0.f;
    if (z1[i] > 0.f) {
        for (int dz = (pz + 1) & 1; dz < 3; dz += 2) {   // the stride of 2: taps of the position's parity
            const int tz = pz + 1 - dz;
            if (tz >= 8) continue;
            for (int dy = (py + 1) & 1; dy < 3; dy += 2) {
                const int ty = py + 1 - dy;
                if (ty >= 8) continue;
                for (int dx = (px + 1) & 1; dx < 3; dx += 2) {
                    const int tx = px + 1 - dx;
                    if (tx >= 8) continue;
                    const int o = (tz / 2 * 4 + ty / 2) * 4 + tx / 2;
                    s += da[((int64_t)b * kP2 + o) * kK2 + c * 27 + dz * 9 + dy * 3 + dx];
                }
            }
        }
    }
    dz1[i] = s;
    dz1b[i] = __float2bfloat16_rn(s);
}
// The first half of db1's column sums: part[t][c] = sum of rows t, t + 256, ... of column c, in that order.
// 16 lanes read a row's 16 columns.
__global__ void __launch_bounds__(256) k_colsum1(const float* __restrict__ x, int64_t rows, float* __restrict__ part) {
    grid_dependency();
    const int t = blockIdx.x * 16 + threadIdx.x / kC1, c = threadIdx.x % kC1;
    float s = 0.f;
#pragma unroll 16
    for (int64_t r = t; r < rows; r += 256) s += x[r * kC1 + c];
    part[t * kC1 + c] = s;
}
// The small gradients and the loss, one block each, in a fixed order.  Block 0: the sum of the squared
// errors; 1: db4; 2 .. 33: dW4; then db3 (32), db2 (16) and db1 (16, from k_colsum1's sums).
constexpr int kSmallBlocks = 2 + 2 * kF + kC2 + kC1;
__global__ void __launch_bounds__(256) k_small_grads(const float* __restrict__ sq, const float* __restrict__ dout,
                                                     const bf16* __restrict__ h3, const float* __restrict__ dz3,
                                                     const float* __restrict__ dz2, const float* __restrict__ part1, int B,
                                                     float* __restrict__ grads, float* __restrict__ loss) {
    grid_dependency();
    const int k = blockIdx.x;
    float s = 0.f;
    if (k >= 1 && k < 2 + kF) {   // one chain over the tiles
        __shared__ float v[2][256];
        for (int b0 = 0; b0 < B; b0 += 256) {
            const int b = b0 + threadIdx.x;
            if (b < B) {
                v[0][threadIdx.x] = dout[b];
                v[1][threadIdx.x] = k == 1 ? 1.f : __bfloat162float(h3[(int64_t)b * kF + (k - 2)]);
            }
            __syncthreads();
            if (threadIdx.x == 0)
                for (int i = 0; i < min(256, B - b0); i++) s = k == 1 ? s + v[0][i] : fmaf(v[1][i], v[0][i], s);
            __syncthreads();
        }
        if (threadIdx.x == 0) grads[k == 1 ? kOffB4 : kOffW4 + (k - 2)] = s;
        return;
    }
    float* dst;
    auto sum = [&](const float* x, int64_t rows, int cols, int c) {
#pragma unroll 8
        for (int64_t r = threadIdx.x; r < rows; r += 256) s += x[r * cols + c];
    };
    if (k == 0) { dst = loss; sum(sq, B, 1, 0); }
    else if (k < 2 + 2 * kF) { dst = grads + kOffB3 + (k - 2 - kF); sum(dz3, B, kF, k - 2 - kF); }
    else if (k < 2 + 2 * kF + kC2) { dst = grads + kOffB2 + (k - 2 - 2 * kF); sum(dz2, (int64_t)B * kP2, kC2, k - 2 - 2 * kF); }
    else { dst = grads + kOffB1 + (k - 2 - 2 * kF - kC2); s = part1[threadIdx.x * kC1 + (k - 2 - 2 * kF - kC2)]; }
    __shared__ float red[256];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *dst = red[0];
}
// Adam on the FP32 master parameters, and the BF16 copies of W1, W2, W3
__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       int64_t n, float lr, float b1, float b2, float eps, float c1, float c2, bf16* __restrict__ wb) {
    grid_dependency();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    constexpr int N1 = kK1 * kC1, N2 = kK2 * kC2;
    const bf16 r = __float2bfloat16_rn(w[i]);
    if (i < N1) wb[i] = r;
    else if (i >= (int)kOffW2 && i < (int)kOffB2) wb[N1 + (i - (int)kOffW2)] = r;
    else if (i >= (int)kOffW3 && i < (int)kOffB3) wb[N1 + N2 + (i - (int)kOffW3)] = r;
}
__global__ void k_to_bf16(const float* __restrict__ x, int64_t n, bf16* __restrict__ y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

inline unsigned blocks(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace

// ------------------------------------------------------------------ the network object
struct Estimator {
    uint32_t max_batch = 0;
    float* params = nullptr;     // FP32 master parameters (kParams)
    float* grads = nullptr;      // FP32 gradients, same layout
    float* adam_m = nullptr;
    float* adam_v = nullptr;
    bf16* wb = nullptr;          // BF16 copies of W1, W2, W3 (GEMM operands)
    // activations and their gradients for max_batch tiles
    bf16 *h1 = nullptr, *h2 = nullptr, *h3 = nullptr;
    float *z1 = nullptr, *z2 = nullptr, *z3 = nullptr, *out = nullptr;
    float *dout = nullptr, *sq = nullptr, *dz3 = nullptr, *dz2 = nullptr, *dz1 = nullptr, *da2 = nullptr, *loss = nullptr;
    bf16 *dz3b = nullptr, *dz2b = nullptr, *dz1b = nullptr;
    Chunk *pa1 = nullptr, *pb1 = nullptr, *pa2 = nullptr, *pb2 = nullptr;   // packed operands of dW1 and dW2
    float* part1 = nullptr;                                                 // db1's column sums, first half
    int step = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t side = nullptr;     // backward()'s work beside the chain of the convolutions' gradients
    cudaEvent_t ev[3] = {};

    ~Estimator() {
        if (stream) cudaStreamSynchronize(stream);
        if (side) cudaStreamSynchronize(side);
        for (void* p : {(void*)params, (void*)grads, (void*)adam_m, (void*)adam_v, (void*)wb, (void*)h1, (void*)h2,
                        (void*)h3, (void*)z1, (void*)z2, (void*)z3, (void*)out, (void*)dout, (void*)sq, (void*)dz3,
                        (void*)dz2, (void*)dz1, (void*)da2, (void*)loss, (void*)dz3b, (void*)dz2b, (void*)dz1b,
                        (void*)pa1, (void*)pb1, (void*)pa2, (void*)pb2, (void*)part1})
            cudaFree(p);
        for (cudaEvent_t x : ev)
            if (x) cudaEventDestroy(x);
        if (side) cudaStreamDestroy(side);
        if (stream) cudaStreamDestroy(stream);
    }
    template <class T>
    static cudaError_t alloc(T** p, size_t n) { return cudaMalloc((void**)p, n * sizeof(T)); }

    cudaError_t init(uint32_t batch, uint64_t seed) {
        max_batch = batch;
        const size_t B = batch;
        cudaError_t e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking);
        for (cudaEvent_t& x : ev)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
        if (e == cudaSuccess) e = alloc(&params, kParams);
        if (e == cudaSuccess) e = alloc(&grads, kParams);
        if (e == cudaSuccess) e = alloc(&adam_m, kParams);
        if (e == cudaSuccess) e = alloc(&adam_v, kParams);
        if (e == cudaSuccess) e = alloc(&wb, (size_t)kK1 * kC1 + (size_t)kK2 * kC2 + (size_t)kK3 * kF);
        if (e == cudaSuccess) e = alloc(&h1, B * kP1 * kC1);
        if (e == cudaSuccess) e = alloc(&h2, B * kK3);
        if (e == cudaSuccess) e = alloc(&h3, B * kF);
        if (e == cudaSuccess) e = alloc(&z1, B * kP1 * kC1);
        if (e == cudaSuccess) e = alloc(&z2, B * kP2 * kC2);
        if (e == cudaSuccess) e = alloc(&z3, B * kF);
        if (e == cudaSuccess) e = alloc(&out, B);
        if (e == cudaSuccess) e = alloc(&dout, B);
        if (e == cudaSuccess) e = alloc(&sq, B);
        if (e == cudaSuccess) e = alloc(&dz3, B * kF);
        if (e == cudaSuccess) e = alloc(&dz2, B * kK3);
        if (e == cudaSuccess) e = alloc(&loss, 1);
        if (e == cudaSuccess) e = alloc(&dz3b, B * kF);
        if (e == cudaSuccess) e = alloc(&dz2b, B * kK3);
        if (e == cudaSuccess) e = alloc(&dz1b, B * kP1 * kC1);
        if (e == cudaSuccess) e = alloc(&dz1, B * kP1 * kC1);
        if (e == cudaSuccess) e = alloc(&da2, B * kP2 * kK2);
        if (e == cudaSuccess) e = alloc(&pa1, B * kP1 * kK1 / 8);
        if (e == cudaSuccess) e = alloc(&pb1, B * kP1 * kC1 / 8);
        if (e == cudaSuccess) e = alloc(&pa2, B * kP2 * kK2 / 8);
        if (e == cudaSuccess) e = alloc(&pb2, B * kP2 * kC2 / 8);
        if (e == cudaSuccess) e = alloc(&part1, 256u * kC1);
        if (e != cudaSuccess) return e;
        // He-uniform initial weights from a seeded 64-bit LCG, zero biases
        std::vector<float> h(kParams, 0.f);
        uint64_t s = seed * 6364136223846793005ull + 1442695040888963407ull;
        auto uni = [&]() {
            s = s * 6364136223846793005ull + 1442695040888963407ull;
            return (float)((double)(s >> 11) * (1.0 / 9007199254740992.0)) * 2.f - 1.f;
        };
        auto fill = [&](size_t off, int rows, int real_rows, int cols, int fan_in) {
            const float a = std::sqrt(6.f / (float)fan_in);
            for (int r = 0; r < rows; r++)
                for (int c = 0; c < cols; c++) h[off + (size_t)r * cols + c] = r < real_rows ? a * uni() : 0.f;
        };
        fill(kOffW1, kK1, kK1Real, kC1, kK1Real);
        fill(kOffW2, kK2, kK2, kC2, kK2);
        fill(kOffW3, kK3, kK3, kF, kK3);
        fill(kOffW4, kF, kF, 1, kF);
        e = set_params(h.data());
        if (e == cudaSuccess) e = cudaMemsetAsync(adam_m, 0, kParams * 4, stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(adam_v, 0, kParams * 4, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        step = 0;
        return e;
    }
    cudaError_t refresh_bf16() {
        k_to_bf16<<<blocks((int64_t)kK1 * kC1), 256, 0, stream>>>(params + kOffW1, (int64_t)kK1 * kC1, wb);
        k_to_bf16<<<blocks((int64_t)kK2 * kC2), 256, 0, stream>>>(params + kOffW2, (int64_t)kK2 * kC2, wb + kK1 * kC1);
        k_to_bf16<<<blocks((int64_t)kK3 * kF), 256, 0, stream>>>(params + kOffW3, (int64_t)kK3 * kF,
                                                                wb + kK1 * kC1 + kK2 * kC2);
        return cudaGetLastError();
    }
    cudaError_t set_params(const float* host) {
        cudaError_t e = cudaMemcpyAsync(params, host, kParams * 4, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = refresh_bf16();
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        return e;
    }

    // forward pass of B tiles (x: device [B][3][512] FP32); predictions in `pred`; with targets, also
    // what backward() needs
    cudaError_t forward(const float* x, int B, const float* target, float* pred) {
        const bf16* W1 = wb;
        const bf16* W2 = wb + kK1 * kC1;
        const bf16* W3 = wb + kK1 * kC1 + kK2 * kC2;
        const int r1 = B * kP1, r2 = B * kP2;
        cudaError_t e = gemm<16, kK1, 2>(Conv1A{x, r1}, WeightB<kC1, kK1>{W1}, BiasRelu<16>{params + kOffB1, target ? z1 : nullptr, h1, r1},
                                 r1, kC1, kK1, stream);
        if (e == cudaSuccess)
            e = gemm<16, kK2, 4>(Conv2A{h1, r2}, WeightB<kC2, kK2>{W2}, BiasRelu<16>{params + kOffB2, target ? z2 : nullptr, h2, r2}, r2, kC2,
                         kK2, stream);
        if (e == cudaSuccess)
            e = gemm<32, kK3, 4>(RowsA<kK3>{h2, B}, WeightB<kF, kK3>{W3}, BiasRelu<32>{params + kOffB3, z3, h3, B}, B, kF, kK3, stream);
        if (e != cudaSuccess) return e;
        return launch_dependent(true, k_fc2, (unsigned)((B + 3) / 4), 128, 0, stream, h3, params + kOffW4, params + kOffB4, B, pred,
                                target, dout, sq, z3, dz3, dz3b);
    }
    // `to` goes on when what `from` holds so far is done
    cudaError_t after(cudaStream_t from, cudaStream_t to, cudaEvent_t x) {
        const cudaError_t e = cudaEventRecord(x, from);
        return e == cudaSuccess ? cudaStreamWaitEvent(to, x, 0) : e;
    }
    // Gradients of the mean squared error of the last forward pass (of x, with targets) into `grads`.  What the
    // convolutions' chain does not need, the dense layer's gradient and the small ones, runs beside it on a
    // stream of its own: a step of 64 tiles, which waits for one chain of MMAs, 244 -> 234 us.
    // (The launches of both passes start while the kernel before drains: 234 -> 215 us.)
    cudaError_t backward(const float* x, int B) {
        const cudaError_t e = backward_passes(x, B);
        const cudaError_t joined = after(side, stream, ev[2]);   // in any case: nothing is left running beside the stream
        return e == cudaSuccess ? joined : e;
    }
    cudaError_t backward_passes(const float* x, int B) {
        const bf16* W2 = wb + kK1 * kC1;
        const bf16* W3 = wb + kK1 * kC1 + kK2 * kC2;
        const int k1 = B * kP1, k2 = B * kP2;
        // dW3 = H2^T dZ3, dH2 = dZ3 W3^T through conv2's ReLU
        cudaError_t e = after(stream, side, ev[0]);
        if (e == cudaSuccess)
            e = gemm<32, 0, 1>(ColumnsT<kK3>{h2, B}, ColumnsT<kF>{dz3b, B}, Store<32, kF>{grads + kOffW3, kK3}, kK3, kF, B, side);
        if (e == cudaSuccess)
            e = gemm<32, kF, 1>(RowsA<kF>{dz3b, B}, RowsA<kF>{W3, kK3}, ReluBack<32, kK3>{z2, dz2, dz2b, B}, B, kK3, kF, stream);
        // dA2 = dY2 W2^T, then col2im through conv1's ReLU
        if (e == cudaSuccess)
            e = gemm<32, kC2, 1>(RowsA<kC2>{dz2b, k2}, RowsA<kC2>{W2, kK2}, Store<32, kK2>{da2, k2}, k2, kK2, kC2, stream);
        if (e != cudaSuccess) return e;
        e = launch_dependent(true, k_col2im2, blocks((int64_t)B * kP1 * kC1), 256, 0, stream, da2, z1, B, dz1, dz1b);
        if (e != cudaSuccess || (e = after(stream, side, ev[1])) != cudaSuccess) return e;
        e = launch_dependent(false, k_colsum1, 16, 256, 0, side, dz1, k1, part1);
        if (e == cudaSuccess)
            e = launch_dependent(true, k_small_grads, kSmallBlocks, 256, 0, side, sq, dout, h3, dz3, dz2, part1, B, grads, loss);
        if (e != cudaSuccess) return e;
        // dW1 = A1^T dY1 (rows 81..95 of A1 are zero, so their gradient is too) and dW2 = A2^T dY2
        const int64_t chunks = (int64_t)(kK1 + 16) * (k1 / kGemmK) * 8 + (int64_t)(kK2 + 16) * (k2 / kGemmK) * 8;
        e = launch_dependent(false, k_pack<Conv1At, ColumnsT<kC1>, Conv2At, ColumnsT<kC2>>, blocks(chunks), 256, 0, stream, Conv1At{x},
                             ColumnsT<kC1>{dz1b, k1}, kK1, k1, pa1, pb1, Conv2At{h1}, ColumnsT<kC2>{dz2b, k2}, kK2, k2, pa2, pb2);
        if (e != cudaSuccess) return e;
        int* err = device_error_flag();
        if (!err) return cudaErrorMemoryAllocation;
        static std::atomic<uint64_t> configured{0};
        if ((e = ensure_smem_limit(k_stream_gemm, kStreamSmem, configured)) != cudaSuccess) return e;
        return launch_dependent(true, k_stream_gemm, (kK1 + kK2) / kSlabRows, 64, kStreamSmem, stream,
                                StreamGemm{pa1, pb1, grads + kOffW1, kK1, k1 / kGemmK},
                                StreamGemm{pa2, pb2, grads + kOffW2, kK2, k2 / kGemmK}, err);
    }
    cudaError_t adam(float lr) {
        step++;
        const float b1 = .9f, b2 = .999f;
        k_adam<<<blocks((int64_t)kParams), 256, 0, stream>>>(params, grads, adam_m, adam_v, (int64_t)kParams, lr, b1, b2,
                                                            1e-8f, 1.f - std::pow(b1, (float)step),
                                                            1.f - std::pow(b2, (float)step), wb);
        return cudaGetLastError();
    }
};

size_t estimator_param_count() { return kParams; }

}  // namespace amr

using namespace amr;

#define AMR_API extern "C" __attribute__((visibility("default")))

struct amr_estimator {
    Estimator net;
};

AMR_API int amr_estimator_create(uint32_t max_batch, uint64_t seed, amr_estimator** out) {
    if (!out || max_batch == 0 || max_batch > (1u << 16)) return AMR_ERR_INVALID;
    amr_estimator* e = new (std::nothrow) amr_estimator;
    if (!e) return AMR_ERR_CAPACITY;
    const cudaError_t st = e->net.init(max_batch, seed);
    if (st != cudaSuccess) {
        delete e;
        return cuda_status(st);
    }
    *out = e;
    return AMR_OK;
}
AMR_API int amr_estimator_destroy(amr_estimator* e) {
    delete e;
    return AMR_OK;
}
AMR_API uint64_t amr_estimator_param_count(void) { return kParams; }
AMR_API int amr_estimator_get_params(amr_estimator* e, float* host) {
    if (!e || !host) return AMR_ERR_INVALID;
    cudaError_t st = cudaMemcpyAsync(host, e->net.params, kParams * 4, cudaMemcpyDeviceToHost, e->net.stream);
    if (st == cudaSuccess) st = cudaStreamSynchronize(e->net.stream);
    return cuda_status(st);
}
AMR_API int amr_estimator_set_params(amr_estimator* e, const float* host) {
    if (!e || !host) return AMR_ERR_INVALID;
    return cuda_status(e->net.set_params(host));
}
AMR_API int amr_estimator_forward(amr_estimator* e, const float* features, uint32_t n, float* out) {
    if (!e || (n && (!features || !out))) return AMR_ERR_INVALID;
    for (uint32_t b0 = 0; b0 < n; b0 += e->net.max_batch) {
        const int B = (int)std::min<uint32_t>(e->net.max_batch, n - b0);
        const cudaError_t st = e->net.forward(features + (size_t)b0 * kIn * kP1, B, nullptr, out + b0);
        if (st != cudaSuccess) return cuda_status(st);
    }
    const int st = cuda_status(cudaStreamSynchronize(e->net.stream));
    return st ? st : take_device_error(device_error_flag());
}
AMR_API int amr_estimator_gradients(amr_estimator* e, const float* features, const float* targets, uint32_t n,
                                    float* grads_host, float* loss) {
    if (!e || !features || !targets || n == 0 || n > e->net.max_batch) return AMR_ERR_INVALID;
    cudaError_t st = e->net.forward(features, (int)n, targets, e->net.out);
    if (st == cudaSuccess) st = e->net.backward(features, (int)n);
    float l = 0.f;
    if (st == cudaSuccess && grads_host)
        st = cudaMemcpyAsync(grads_host, e->net.grads, kParams * 4, cudaMemcpyDeviceToHost, e->net.stream);
    if (st == cudaSuccess) st = cudaMemcpyAsync(&l, e->net.loss, 4, cudaMemcpyDeviceToHost, e->net.stream);
    if (st == cudaSuccess) st = cudaStreamSynchronize(e->net.stream);
    if (loss) *loss = l / (float)n;
    const int status = cuda_status(st);
    return status ? status : take_device_error(device_error_flag());
}
AMR_API int amr_estimator_train_step(amr_estimator* e, const float* features, const float* targets, uint32_t n,
                                     float lr, float* loss) {
    if (!e || !features || !targets || n == 0 || n > e->net.max_batch || !(lr > 0.f)) return AMR_ERR_INVALID;
    cudaError_t st = e->net.forward(features, (int)n, targets, e->net.out);
    if (st == cudaSuccess) st = e->net.backward(features, (int)n);
    if (st == cudaSuccess) st = e->net.adam(lr);
    float l = 0.f;
    if (st == cudaSuccess && loss) st = cudaMemcpyAsync(&l, e->net.loss, 4, cudaMemcpyDeviceToHost, e->net.stream);
    if (st == cudaSuccess) st = cudaStreamSynchronize(e->net.stream);
    if (loss) *loss = l / (float)n;
    const int status = cuda_status(st);
    return status ? status : take_device_error(device_error_flag());
}
