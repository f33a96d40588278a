// kernels_point.cu -- cell-local kernels (one thread per interior cell or codec word).
#include "kernels.h"

#include "amr_device.cuh"

namespace amr {

namespace {

constexpr int kBlock = 256;

inline uint32_t blocks_for(uint64_t n) { return (uint32_t)((n + kBlock - 1) / kBlock); }

// A thread's cell: its domain, inner-layout index o and padded index.  A block's cells lie in one domain
// (domain_blocks blocks each) of a compiled size, so that no index is divided in 64 bits or by a variable:
// the pointwise kernels were bound by issue (70 % of the slots), their trace is now near the copy
// bandwidth (1.08 M cells of 28^3, 10.7 -> 10.1 us; the Christoffel symbols, with encodes in pairs, 25.7 ->
// 23.7).
struct InnerCell {
    uint32_t slot, x, y, z;
    uint64_t o, padded;
};
inline uint32_t domain_blocks(const Dims& d) { return (d.n * d.n * d.n + kBlock - 1) / kBlock; }
template <int N, int P>
__device__ __forceinline__ bool inner_cell(InnerCell& c) {   // false: past the domain's cells
    constexpr uint32_t T = N + 2 * P, n3 = N * N * N, per = (n3 + kBlock - 1) / kBlock;
    c.slot = blockIdx.x / per;
    uint32_t r = (blockIdx.x - c.slot * per) * kBlock + threadIdx.x;
    if (r >= n3) return false;
    c.o = (uint64_t)c.slot * n3 + r;
    c.x = r % N; r /= N;
    c.y = r % N;
    c.z = r / N;
    c.padded = (uint64_t)c.slot * (T * T * T) + ((c.z + P) * T + c.y + P) * T + c.x + P;
    return true;
}
__device__ __forceinline__ bool slot_active(const uint32_t* positions, uint32_t slot, uint32_t substep,
                                            uint32_t max_depth, int* depth_out) {
    const int depth = pos_depth(positions[slot]);
    *depth_out = depth;
    return depth != -1 && active_depth(substep, (uint32_t)depth, max_depth);
}

struct Ptr6f { float* p[6]; };
struct Ptr6u { uint32_t* p[6]; };

// ---------------------------------------------------------------- codec
__global__ void k_cf3_encode(const float* __restrict__ xyz, const int32_t* __restrict__ seeds, uint64_t n,
                             uint32_t* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
    if (seeds) {
        int32_t s = seeds[i];
        out[i] = cf3_encode_codec(x, y, z, s);
    } else {
        out[i] = cf3_encode_det(x, y, z);
    }
}
__global__ void k_cf3_decode(const uint32_t* __restrict__ w, uint64_t n, float* __restrict__ xyz) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float3 v = cf3_decode(w[i]);
    xyz[3 * i] = v.x; xyz[3 * i + 1] = v.y; xyz[3 * i + 2] = v.z;
}

// ---------------------------------------------------------------- g^kl H_kl, BSSN.h:7-22
template <int N, int P>
__global__ void k_deriv_trace(const uint32_t* __restrict__ hd, const uint32_t* __restrict__ ho, Ptr6f m,
                              float* __restrict__ out, const uint32_t* __restrict__ positions, uint32_t substep,
                              uint32_t max_depth) {
    InnerCell c;
    if (!inner_cell<N, P>(c)) return;
    const uint64_t o = c.o;
    int depth;
    if (!slot_active(positions, c.slot, substep, max_depth, &depth)) return;
    const Sym g{m.p[0][c.padded], m.p[1][c.padded], m.p[2][c.padded], m.p[3][c.padded], m.p[4][c.padded], m.p[5][c.padded]};
    out[o] = trace_contra(sym_from_cf3(hd[o], ho[o]), sym_inverse(g));
}

// ---------------------------------------------------------------- Christoffel symbols, BSSN.h:55-91
template <int N, int P>
__global__ void k_christoffel(Ptr6f m, Ptr6u der, int32_t seed, Ptr6u outp,
                              const uint32_t* __restrict__ positions, uint32_t substep, uint32_t max_depth,
                              int mode) {
    InnerCell c;
    if (!inner_cell<N, P>(c)) return;
    const uint64_t o = c.o;
    int depth;
    if (!slot_active(positions, c.slot, substep, max_depth, &depth)) return;
    int32_t rng = cell_rng(seed, c.x, c.y, c.slot * N + c.z);
    uint32_t G[6];
#pragma unroll
    for (int k = 0; k < 6; k++) G[k] = der.p[k][o];
    const Sym g{m.p[0][c.padded], m.p[1][c.padded], m.p[2][c.padded], m.p[3][c.padded], m.p[4][c.padded], m.p[5][c.padded]};
    const Sym M = mode == AMR_CHRISTOFFEL_RAISED ? sym_inverse(g) : g;
    float2 noise[9];
#pragma unroll
    for (int k = 0; k < 3; k++) noise_pairs1(rng, noise[3 * k], noise[3 * k + 1], noise[3 * k + 2]);
    uint32_t out[6];
    christoffel_cell(G, M, noise, out);
#pragma unroll
    for (int jk = 0; jk < 6; jk++) outp.p[jk][o] = out[jk];
}

// ---------------------------------------------------------------- SimpleWave Heun update, SimpleWave.h:7-46
template <int N, int P>
__global__ void k_wave_step(float outer_dt, int corrector, const float* __restrict__ old_f,
                            const uint32_t* __restrict__ der, const uint32_t* __restrict__ hess, float* new_f,
                            const uint32_t* __restrict__ positions, uint32_t substep, uint32_t max_depth) {
    grid_dependency();
    InnerCell c;
    if (!inner_cell<N, P>(c)) return;
    const uint64_t o = c.o;
    int depth;
    if (!slot_active(positions, c.slot, substep, max_depth, &depth)) return;
    const float w = wave_update(old_f[c.padded], cf3_decode(der[o]).x, cf3_decode(hess[o]), outer_dt, depth);
    new_f[c.padded] = corrector ? __fmul_rn(__fadd_rn(new_f[c.padded], w), .5f) : w;
}

// ---------------------------------------------------------------- refinement criterion, SimpleWave.h:91-139
__device__ __forceinline__ float cf3_length(uint32_t w) {
    const float3 v = cf3_decode(w);
    return sqrt_approx(__fmaf_rn(v.z, v.z, __fmaf_rn(v.x, v.x, __fmul_rn(v.y, v.y))));
}
// A CTA per octant.  The reference's first kernel writes a column's largest value for each column of the
// octant (its h cells along z in the octant, of rows y and y + q), the second the octant's maximum over
// them, in order from NaN, to its first column's place (SimpleWave.h:91-139).  The values are non-negative
// or NaN and fmaxf skips NaN, so the maxima do not depend on the order: `parts` threads share a column.
// (A thread per column and a second launch took 12.5 + 4.0 us on 9 domains of 28^3, a chain of 14 loads; this 6.2.)
constexpr uint32_t kCritThreads = 512;
__global__ void __launch_bounds__(kCritThreads) k_criterion(Dims d, float outer_dx, const uint32_t* __restrict__ der,
                                                           const uint32_t* __restrict__ hess, float* __restrict__ crit,
                                                           const uint32_t* __restrict__ positions, uint32_t substep,
                                                           uint32_t max_depth) {
    const uint32_t n = d.n, h = n >> 1, q = n >> 2, columns = q * h;
    grid_dependency();
    const uint32_t oct = blockIdx.x & 7u, node = blockIdx.x >> 3;
    const uint32_t xb = oct & 1u, yb = (oct >> 1) & 1u, zi = 2u * node + (oct >> 2);
    const uint64_t base = ((uint64_t)zi * h + yb * q) * n + xb * h;
    const int depth = pos_depth(positions[node]);
    if (depth == -1 || !active_depth(substep, (uint32_t)depth, max_depth)) {   // NAN, SimpleWave.h:97
        for (uint32_t c = threadIdx.x; c < columns; c += kCritThreads) crit[base + c % h + (uint64_t)(c / h) * n] = __int_as_float(0x7fc00000);
        return;
    }
    // |g| * dx / 2^depth and |H| * dx * dx / 4^depth, left to right (the power-of-two scaling is exact)
    const float s1 = __uint_as_float((127u - (uint32_t)depth) << 23);
    const float s2 = __uint_as_float((127u - 2u * (uint32_t)depth) << 23);
    __shared__ float part[kCritThreads];
    const uint32_t parts = min(h, kCritThreads / columns);   // at least 2 (16^3: 16; 32^3: 4)
    const uint32_t c = threadIdx.x % columns, k = threadIdx.x / columns;
    float cr = 0.f;
    if (k < parts) {
        const uint32_t x = xb * h + c % h, y = c / h + (yb ? 2u * q : 0u);
        const uint64_t ro = x + ((uint64_t)y + (uint64_t)zi * n * h) * n;
        for (uint32_t i = k; i < h; i += parts) {
            const uint64_t r0 = ro + (uint64_t)i * n * n, r1 = r0 + (uint64_t)q * n;
            cr = fmaxf(cr, __fmul_rn(__fmul_rn(cf3_length(der[r0]), outer_dx), s1));
            cr = fmaxf(cr, __fmul_rn(__fmul_rn(__fmul_rn(cf3_length(hess[r0]), outer_dx), outer_dx), s2));
            cr = fmaxf(cr, __fmul_rn(__fmul_rn(cf3_length(der[r1]), outer_dx), s1));
            cr = fmaxf(cr, __fmul_rn(__fmul_rn(__fmul_rn(cf3_length(hess[r1]), outer_dx), outer_dx), s2));
        }
    }
    part[threadIdx.x] = cr;
    __syncthreads();
    if (k == 0) {
        for (uint32_t j = 1; j < parts; j++) cr = fmaxf(cr, part[threadIdx.x + j * columns]);
        if (c != 0) crit[base + c % h + (uint64_t)(c / h) * n] = cr;
        part[threadIdx.x] = cr;
    }
    __syncthreads();
    if (threadIdx.x < 32u) {
        cr = __int_as_float(0x7fc00000);
        for (uint32_t e = threadIdx.x; e < columns; e += 32u) cr = fmaxf(cr, part[e]);
#pragma unroll
        for (int s = 16; s >= 1; s >>= 1) cr = fmaxf(cr, __shfl_xor_sync(0xFFFFFFFFu, cr, s));
        if (threadIdx.x == 0) crit[base] = cr;
    }
}

// ---------------------------------------------------------------- slice rasteriser, AMR.h:1313-1352
// One thread per pixel of a z-slice through the unit cube: descend the octree to the leaf holding
// the point, interpolate the padded field there (10-point, AMR.h:672-699) and write grey RGBA, or
// red near the leaf's border when bounding boxes are drawn (the reference's build draws them).
// As the reference's fast-math build computes them, px / width - 0.5 is a fused multiply-add with
// the approximate reciprocal of width, and so is the border threshold.  The descent stops at
// kDepthLimit levels or at a child index outside the used slots.
__global__ void k_rasterise(Dims d, const float* __restrict__ data, const int32_t* __restrict__ children,
                            uint32_t used, uint32_t width, uint32_t height, float z_slice, int boxes,
                            float4* __restrict__ raster) {
    const uint32_t px = blockIdx.x * blockDim.x + threadIdx.x, py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= width || py >= height) return;
    const float rw = rcp_approx((float)width), rh = rcp_approx((float)height);
    float tp[3] = {__fmaf_rn((float)px, rw, -.5f), __fmaf_rn((float)py, rh, -.5f), z_slice};
    auto octant = [&]() { return (uint32_t)(tp[0] > 0.f) | ((uint32_t)(tp[1] > 0.f) << 1) | ((uint32_t)(tp[2] > 0.f) << 2); };
    uint32_t curr = 0, depth = 0;
    int32_t child = children[octant()];
    for (; child != -1 && (uint32_t)child < used && depth < kDepthLimit; depth++) {
        curr = (uint32_t)child;
#pragma unroll
        for (int a = 0; a < 3; a++) {   // fracf(2 t) - 0.5, helper_math.h:1475-1478
            const float v = __fmul_rn(tp[a], 2.f);
            tp[a] = __fsub_rn(__fsub_rn(v, floorf(v)), .5f);
        }
        child = children[curr * 8u + octant()];
    }
    if (boxes) {   // DISPLAY_BOUNDING_BOXES (AMR.h:1312, 1329-1337): red where the leaf's border is near
        const float threshold = __fmaf_rn(-__fmul_rn(2.f, (float)(1u << depth)), rw, .5f);
        if (fmaxf(fabsf(tp[0]), fabsf(tp[1])) >= threshold) {
            raster[(size_t)py * width + px] = make_float4(1.f, 0.f, 0.f, 1.f);
            return;
        }
    }
    uint32_t ri[3];
    float r[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float q = __fmaf_rn(__fadd_rn(tp[a], .5f), (float)d.n, (float)d.p);
        ri[a] = __float2uint_rz(__fadd_rn(q, .5f));
        r[a] = __fsub_rn(q, (float)ri[a]);
    }
    const uint64_t rin = (((uint64_t)curr * d.t + ri[2]) * d.t + ri[1]) * d.t + ri[0];
    const float v = __fadd_rn(interp10_strided(data + rin, (int)d.t, (int)(d.t * d.t), r[0], r[1], r[2]), .5f);
    raster[(size_t)py * width + px] = make_float4(v, v, v, 1.f);
}

}  // namespace

// ---------------------------------------------------------------- launchers
cudaError_t launch_cf3_encode(const float* xyz, const int32_t* seeds, uint64_t n, uint32_t* out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_cf3_encode<<<blocks_for(n), kBlock, 0, st>>>(xyz, seeds, n, out);
    return cudaGetLastError();
}
cudaError_t launch_cf3_decode(const uint32_t* w, uint64_t n, float* xyz, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_cf3_decode<<<blocks_for(n), kBlock, 0, st>>>(w, n, xyz);
    return cudaGetLastError();
}
cudaError_t launch_deriv_trace(Dims d, const uint32_t* hd, const uint32_t* ho, float* const* metric6, float* out,
                               const uint32_t* positions, uint32_t used, uint32_t substep, uint32_t max_depth,
                               cudaStream_t st) {
    if (used == 0) return cudaSuccess;
    Ptr6f m;
    for (int k = 0; k < 6; k++) m.p[k] = metric6[k];
#define AMR_POINT(N, P) \
    if (d.n == N && d.p == P) { k_deriv_trace<N, P><<<used * domain_blocks(d), kBlock, 0, st>>>(hd, ho, m, out, positions, substep, max_depth); return cudaGetLastError(); }
    AMR_FOR_EACH_CONFIG(AMR_POINT)
#undef AMR_POINT
    return cudaErrorInvalidValue;
}
cudaError_t launch_christoffel(Dims d, float* const* metric6, uint32_t* const* der6, int32_t seed, uint32_t* const* out6,
                               const uint32_t* positions, uint32_t used, uint32_t substep, uint32_t max_depth, int mode,
                               cudaStream_t st) {
    if (used == 0) return cudaSuccess;
    Ptr6f m; Ptr6u der, out;
    for (int k = 0; k < 6; k++) { m.p[k] = metric6[k]; der.p[k] = der6[k]; out.p[k] = out6[k]; }
#define AMR_POINT(N, P) \
    if (d.n == N && d.p == P) { k_christoffel<N, P><<<used * domain_blocks(d), kBlock, 0, st>>>(m, der, seed, out, positions, substep, max_depth, mode); return cudaGetLastError(); }
    AMR_FOR_EACH_CONFIG(AMR_POINT)
#undef AMR_POINT
    return cudaErrorInvalidValue;
}
cudaError_t launch_wave_step(Dims d, const Geo& g, int corrector, const float* old_f, const uint32_t* der,
                             const uint32_t* hess, float* new_f, const uint32_t* positions, uint32_t used,
                             uint32_t substep, uint32_t max_depth, cudaStream_t st, bool early) {
    if (used == 0) return cudaSuccess;
#define AMR_POINT(N, P) \
    if (d.n == N && d.p == P) { \
        return launch_dependent(early, k_wave_step<N, P>, used * domain_blocks(d), kBlock, 0, st, g.outer_dt, corrector, old_f, der,    \
                                hess, new_f, positions, substep, max_depth); }
    AMR_FOR_EACH_CONFIG(AMR_POINT)
#undef AMR_POINT
    return cudaErrorInvalidValue;
}
cudaError_t launch_criterion(Dims d, const Geo& g, const uint32_t* der, const uint32_t* hess, float* crit,
                             const uint32_t* positions, uint32_t used, uint32_t substep, uint32_t max_depth,
                             cudaStream_t st, bool early) {
    if (used == 0) return cudaSuccess;
    if (d.n < 4u || (d.n >> 1) * (d.n >> 2) > kCritThreads) return cudaErrorInvalidValue;
    return launch_dependent(early, k_criterion, used * 8u, kCritThreads, 0, st, d, g.outer_dx, der, hess, crit, positions, substep,
                            max_depth);
}

cudaError_t launch_rasterise(Dims d, const float* data, const int32_t* children, uint32_t used, uint32_t width,
                             uint32_t height, float z_slice, int boxes, float* raster, cudaStream_t st) {
    if (width == 0 || height == 0) return cudaSuccess;
    const dim3 threads(32, 8), grid((width + 31) / 32, (height + 7) / 8);
    k_rasterise<<<grid, threads, 0, st>>>(d, data, children, used, width, height, z_slice, boxes,
                                          reinterpret_cast<float4*>(raster));
    return cudaGetLastError();
}

// ---------------------------------------------------------------- words carried by a launch
namespace {
struct WordBlock {
    static constexpr uint32_t kMax = 1000;   // 4 KB of parameters
    int32_t v[kMax];
    uint32_t n;
};
__global__ void k_store_words(int32_t* __restrict__ dst, const __grid_constant__ WordBlock b) {
    for (uint32_t i = threadIdx.x; i < b.n; i += blockDim.x) dst[i] = b.v[i];
}
}  // namespace

cudaError_t launch_store_words(int32_t* dst, const int32_t* words, uint32_t n, cudaStream_t st, uint32_t* launched) {
    uint32_t count = 0;
    for (uint32_t at = 0; at < n; at += WordBlock::kMax) {
        WordBlock b;
        b.n = n - at < WordBlock::kMax ? n - at : WordBlock::kMax;
        for (uint32_t i = 0; i < b.n; i++) b.v[i] = words[at + i];
        k_store_words<<<1, 256, 0, st>>>(dst + at, b);
        count++;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) { if (launched) *launched = count; return e; }
    }
    if (launched) *launched = count;
    return cudaSuccess;
}

// ---------------------------------------------------------------- device-to-device copy
namespace {
// n4 float4 with four loads in flight per thread, then the n % 4 trailing words
__global__ void __launch_bounds__(kBlock) k_copy_words4(float4* __restrict__ dst, const float4* __restrict__ src,
                                                       uint64_t n4, float* __restrict__ dtail,
                                                       const float* __restrict__ stail, uint32_t ntail) {
    const uint64_t stride = (uint64_t)gridDim.x * kBlock;
    uint64_t i = (uint64_t)blockIdx.x * kBlock + threadIdx.x;
    for (; i + 3 * stride < n4; i += 4 * stride) {
        const float4 a = __ldcs(src + i), b = __ldcs(src + i + stride), c = __ldcs(src + i + 2 * stride),
                     d = __ldcs(src + i + 3 * stride);
        __stcs(dst + i, a); __stcs(dst + i + stride, b); __stcs(dst + i + 2 * stride, c); __stcs(dst + i + 3 * stride, d);
    }
    for (; i < n4; i += stride) __stcs(dst + i, __ldcs(src + i));
    if (blockIdx.x == 0 && threadIdx.x < ntail) dtail[threadIdx.x] = stail[threadIdx.x];
}
__global__ void __launch_bounds__(kBlock) k_copy_words1(float* __restrict__ dst, const float* __restrict__ src, uint64_t n) {
    for (uint64_t i = (uint64_t)blockIdx.x * kBlock + threadIdx.x; i < n; i += (uint64_t)gridDim.x * kBlock) dst[i] = src[i];
}
}  // namespace

cudaError_t launch_copy_words(void* dst, const void* src, uint64_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    int dev = 0, sms = 0;   // the current device's
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
    const uint32_t cap = (uint32_t)sms * 8u;
    if ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) % 16u == 0u) {
        const uint64_t n4 = n / 4u;
        const uint32_t want = (uint32_t)((n4 + 4u * kBlock - 1u) / (4u * kBlock));
        const uint32_t grid = want < 1u ? 1u : (want < cap ? want : cap);
        k_copy_words4<<<grid, kBlock, 0, st>>>(static_cast<float4*>(dst), static_cast<const float4*>(src), n4,
                                              static_cast<float*>(dst) + n4 * 4u,
                                              static_cast<const float*>(src) + n4 * 4u, (uint32_t)(n % 4u));
    } else {
        const uint32_t want = blocks_for(n);
        k_copy_words1<<<want < cap ? want : cap, kBlock, 0, st>>>(static_cast<float*>(dst), static_cast<const float*>(src), n);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------- many copies in one launch
namespace {
// blockIdx.y: the copy; its CTAs stride over its 16-byte vectors, then its last n % 4 words
__global__ void __launch_bounds__(kBlock) k_copy_many(const __grid_constant__ CopyList l) {
    const CopyList::Item& it = l.item[blockIdx.y];
    const uint64_t n4 = it.n / 4u;
    const float4* __restrict__ s4 = static_cast<const float4*>(it.src);
    float4* __restrict__ d4 = static_cast<float4*>(it.dst);
    for (uint64_t i = (uint64_t)blockIdx.x * kBlock + threadIdx.x; i < n4; i += (uint64_t)gridDim.x * kBlock)
        __stcs(d4 + i, __ldcs(s4 + i));
    if (blockIdx.x == 0 && threadIdx.x < (uint32_t)(it.n % 4u))
        static_cast<float*>(it.dst)[n4 * 4u + threadIdx.x] = static_cast<const float*>(it.src)[n4 * 4u + threadIdx.x];
}
}  // namespace

cudaError_t launch_copy_many(const CopyList& l, cudaStream_t st) {
    if (l.n == 0) return cudaSuccess;
    if (l.n > CopyList::kMax) return cudaErrorInvalidValue;
    uint64_t most = 0;
    for (uint32_t i = 0; i < l.n; i++) {
        if ((reinterpret_cast<uintptr_t>(l.item[i].dst) | reinterpret_cast<uintptr_t>(l.item[i].src)) % 16u != 0u)
            return cudaErrorInvalidValue;   // the callers' buffers are allocations: 256-byte aligned
        most = l.item[i].n > most ? l.item[i].n : most;
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
    // about 8 CTAs per SM in all, and no more per copy than its largest member's vectors need
    uint64_t per = ((uint64_t)sms * 8u + l.n - 1u) / l.n;
    const uint64_t need = (most / 4u + 4u * kBlock - 1u) / (4u * kBlock);
    per = per < need ? per : need;
    k_copy_many<<<dim3((uint32_t)(per < 1u ? 1u : per), l.n), kBlock, 0, st>>>(l);
    return cudaGetLastError();
}

}  // namespace amr
