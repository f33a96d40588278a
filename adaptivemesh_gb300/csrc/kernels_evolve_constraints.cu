// kernels_evolve_constraints.cu -- Hamiltonian and momentum constraints of the BSSN evolution in one
// kernel, and their norms in double precision.
//
// The constraints need 63 derivatives a cell, of 17 fields.  A pass that stores derivatives (with those
// that only the evolution needs, 111 planes) and a second one that reads them back move ten times the
// bytes of the fields.  Here a persistent CTA takes a tile of one domain, one cell a thread; the fields'
// padded tiles come through a ring of shared-memory slots by bulk copies, requested several fields (and
// into the next tile) ahead, and each thread keeps its cell's derivatives in a column of shared memory,
// where the constraints read them.
//
// Measured on a GB300, 1.08 M cells of 16^3 domains: 139 + 78 us for the two passes, 151 us now (160 with a
// CTA per tile, whose first copies nothing hides); the norms 70 + 107 -> 25 + 8 us.  What bounds it:
// instruction issue (61 % of the slots, 50 % of the shared-memory pipe), about 3 000 instructions a warp.
//
// Compiled with contraction on, as kernels_evolve.cu; H is a difference of large terms, so the
// derivatives and the algebra keep their order of operations.
#include "amr_device.cuh"
#include "evolve.h"
#include "evolve_kernels.h"
#include "evolve_physics.cuh"
#include "kernels.h"
#include "tma.cuh"

namespace amr {

namespace {

constexpr int kConsFields = F_GAMZ + 1;   // chi, gt_ij, K, At_ij, Gt^i: the first 17, in the state's order

// A tile of N x TY x TZ interior cells of one domain, a cell a thread.
template <int N, int TY, int TZ, int R_, int MINB>
struct ConsShape {
    static constexpr int T = N + 6, CT = N * TY * TZ, WARPS = CT / 32;
    static constexpr int PLANES = TZ + 6, CHUNK = (TY + 6) * T;
    static constexpr bool WHOLE = TY == N;               // whole planes: a field's tile is one copy
    // plane pitch of part planes: at 16^3 the half warps take cells a plane apart, whose banks must lie 16 apart
    static constexpr int pitch() {
        int p = CHUNK;
        if (!WHOLE && N == 16) while (p % 32 != 16) p += 4;
        return p;
    }
    static constexpr int PP = pitch(), SLOT = PLANES * PP;
    // ring slots, and how many visits ahead a field is requested: two less than the slots, so that the
    // slot to be refilled was released two visits ago by all but the slowest warps
    static constexpr int R = R_, AHEAD = R - 2;
    static constexpr int COPIES = WHOLE ? 1 : PLANES;
    static constexpr uint32_t COPY_BYTES = 4u * (WHOLE ? SLOT : CHUNK);
    static constexpr int TILES = (N / TY) * (N / TZ);
    static constexpr size_t SMEM = ((size_t)R * SLOT + (size_t)BSSN_ND * CT) * 4u + 2u * R * 8u;
    static_assert(CT % 32 == 0 && N % TY == 0 && N % TZ == 0 && COPIES <= 32 && AHEAD >= 1, "whole warps and tiles");
    static_assert((CHUNK * 4) % 16 == 0 && (TY * T * 4) % 16 == 0 && (T * T * 4) % 16 == 0 && PP % 4 == 0 &&
                  (SLOT * 4) % 16 == 0, "every copy is aligned");
    static_assert(SMEM <= 227u * 1024u && MINB * (SMEM + 1024u) <= 228u * 1024u, "fits an SM");
};

template <int N, int TY, int TZ, int R_, int MINB>
__global__ void __launch_bounds__(ConsShape<N, TY, TZ, R_, MINB>::CT, MINB)
    k_evo_constraints(const __grid_constant__ EvoArgs a, const __grid_constant__ ConsPtrs cons) {
    using S = ConsShape<N, TY, TZ, R_, MINB>;
    constexpr int T = S::T, PP = S::PP, R = S::R, CT = S::CT;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* ring = reinterpret_cast<float*>(smem_raw);
    float* const my = ring + (size_t)R * S::SLOT + threadIdx.x;   // this thread's column
    uint64_t* full = reinterpret_cast<uint64_t*>(ring + (size_t)R * S::SLOT + (size_t)BSSN_ND * CT);
    uint64_t* empty = full + R;
    __shared__ volatile int s_abort;
    __shared__ uint32_t s_asked;   // visits requested
    const uint32_t tid = threadIdx.x, warp = tid / 32u, lane = tid % 32u;
    if (tid == 0) {
        for (int r = 0; r < R; r++) { mbar_init(&full[r], 1); mbar_init(&empty[r], S::WARPS); }
        mbar_fence_init();
        s_abort = 0;
        s_asked = 0;
    }
    grid_dependency();
    __syncthreads();
    const uint32_t tiles = a.n_items * (uint32_t)S::TILES;
    bool ok = true;
    // Request field f's tile t (of domain `slot`), the q-th visit of this CTA, by one whole warp, once every
    // warp has released the slot's previous contents: planes z0 .. z0 + PLANES - 1 and rows y0 .. y0 + TY + 5
    // of the padded domain, a copy per lane.
    auto request = [&](uint32_t q, uint32_t t, uint32_t slot, int f) {
        if (t >= tiles) return;
        const uint32_t s = q % R;
        if (q >= (uint32_t)R) ok = mbar_wait(&empty[s], ((q / R) - 1u) & 1u) && ok;
        if (!__all_sync(0xffffffffu, ok)) return;
        if (lane == 0) {
            mbar_arrive_expect_tx(&full[s], S::COPIES * S::COPY_BYTES);
            atomicMax(&s_asked, q + 1u);   // the warps' requests may pass one another
        }
        __syncwarp();
        const uint32_t k = t % S::TILES, z0 = (k / (N / TY)) * TZ, y0 = (k % (N / TY)) * TY;
        if (lane < (uint32_t)S::COPIES)
            bulk_g2s(ring + (size_t)s * S::SLOT + (size_t)lane * PP,
                     a.fields[f] + ((size_t)slot * T + z0 + lane) * T * T + (size_t)y0 * T, S::COPY_BYTES, &full[s]);
    };
    uint32_t nslot = a.items[blockIdx.x / S::TILES];   // the next tile's slot
    if (warp == 0)
        for (int i = 0; i < S::AHEAD; i++) request(i, blockIdx.x, nslot, i);   // AHEAD <= kConsFields

    const uint32_t x = tid % N;
    uint32_t r = tid / N, zl, y;
    if constexpr (S::WHOLE && N == 16) {   // half warps 8 rows apart: 176 floats = 16 banks
        y = ((r >> 1) & 7u) | ((r & 1u) << 3);
        zl = r >> 4;
    } else if constexpr (S::WHOLE && N == 8 && TZ == 8) {   // quarter warps 2 planes (392 floats = 8 banks) apart
        zl = 2u * (r & 3u) + ((r >> 2) & 1u);
        y = r >> 3;
    } else {
        zl = r % TZ;
        y = r / TZ;
    }
    const int c0 = (int)(zl + 3) * PP + (int)(y + 3) * T + (int)x + 3;
    // the cell's metric, stored form, of the next tile
    float own[6];
    uint32_t npi = 0, nii = 0;
    int ndepth = 0;
    auto load_own = [&](uint32_t t) {   // of tile t, in domain nslot
        const uint32_t k = t % S::TILES, z = (k / (N / TY)) * TZ + zl, yy = (k % (N / TY)) * TY + y;
        npi = (nslot * T + z + 3) * T * T + (yy + 3) * T + x + 3;
        nii = (nslot * N + z) * N * N + yy * N + x;
        ndepth = pos_depth(a.positions[nslot]);
#pragma unroll
        for (int c = 0; c < 6; c++) own[c] = a.fields[F_GXX + c][npi];
    };
    load_own(blockIdx.x);   // the grid has no more CTAs than tiles
    uint32_t v = 0;   // visits consumed
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t pi = npi, ii = nii, slot = nslot;
        const int depth = ndepth;
        if (t + gridDim.x < tiles) nslot = a.items[(t + gridDim.x) / S::TILES];
        const float h = a.prm.outer_size / ((float)N * (float)(1u << depth));
        const float i12h = 1.f / (12.f * h), i12h2 = 1.f / (12.f * h * h), i144h2 = 1.f / (144.f * h * h);
        float u[BSSN_NF];
        float gi[6];   // the inverse conformal metric: xx yy zz xy xz yz
        {
            float m[3][3];
#pragma unroll
            for (int c = 0; c < 6; c++) u[F_GXX + c] = own[c] + bssn_offset(F_GXX + c);   // the stored form is less its offset
            inverse_sym(u + F_GXX, m);
            gi[0] = m[0][0]; gi[1] = m[1][1]; gi[2] = m[2][2];
            gi[3] = m[0][1]; gi[4] = m[0][2]; gi[5] = m[1][2];
        }
        constexpr int st[3] = {1, T, PP};
        // first derivatives into columns d .. d + 2
        auto gradient = [&](const float* q, int d) {
#pragma unroll
            for (int ax = 0; ax < 3; ax++) {
                const int s = st[ax];
                my[(d + ax) * CT] = ((q[-2 * s] - q[2 * s]) + 8.f * (q[s] - q[-s])) * i12h;
            }
        };
        // all six second derivatives: xx yy zz xy xz yz
        auto hessian = [&](const float* q, float* d2) {
#pragma unroll
            for (int ax = 0; ax < 3; ax++) {
                const int s = st[ax];
                d2[ax] = (16.f * (q[-s] + q[s]) - (q[-2 * s] + q[2 * s]) - 30.f * q[0]) * i12h2;
            }
            constexpr int pa[3] = {0, 0, 1}, pb[3] = {1, 2, 2};
            constexpr float w[4] = {1.f, -8.f, 8.f, -1.f};
            constexpr int off[4] = {-2, -1, 1, 2};
#pragma unroll
            for (int m = 0; m < 3; m++) {
                const int sa = st[pa[m]], sb = st[pb[m]];
                float acc = 0.f;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    float row = 0.f;
#pragma unroll
                    for (int v = 0; v < 4; v++) row = fmaf(w[v], q[off[i] * sa + off[v] * sb], row);
                    acc = fmaf(w[i], row, acc);
                }
                d2[3 + m] = acc * i144h2;
            }
        };
        // the next field: the warps take turns to request the one AHEAD visits on, then wait
        auto visit = [&](int f) {
            if (warp == (uint32_t)f % S::WARPS) {
                const int j = f + S::AHEAD;
                if (j < kConsFields) request(v + S::AHEAD, t, slot, j);
                else request(v + S::AHEAD, t + gridDim.x, nslot, j - kConsFields);
            }
            ok = mbar_wait(&full[v % R], (v / R) & 1u) && ok;
            return ring + (size_t)(v % R) * S::SLOT + c0;
        };
        auto release = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[v % R]);
            v++;
        };
#pragma unroll 1
        for (int f = 0; f <= F_GZZ; f++) {
            const float* q = visit(f);
            float d2[6];
            gradient(q, f == F_CHI ? D_CHI1 : D_G1 + 3 * (f - F_GXX));
            hessian(q, d2);
            release();
            if (f == F_CHI) {
#pragma unroll
                for (int c = 0; c < 6; c++) my[(D_CHI2 + c) * CT] = d2[c];
            } else {   // gt^lm d_l d_m gt_ij
                my[(D_GLAP + f - F_GXX) * CT] = gi[0] * d2[0] + gi[1] * d2[1] + gi[2] * d2[2] +
                                                              2.f * (gi[3] * d2[3] + gi[4] * d2[4] + gi[5] * d2[5]);
            }
        }
        u[F_CHI] = a.fields[F_CHI][pi] + bssn_offset(F_CHI);
#pragma unroll
        for (int f = F_K; f < kConsFields; f++) u[f] = a.fields[f][pi] + bssn_offset(f);
        load_own(t + gridDim.x < tiles ? t + gridDim.x : t);   // past the last tile: this one again, unused
#pragma unroll 1
        for (int f = F_K; f < kConsFields; f++) {
            const float* q = visit(f);
            gradient(q, f == F_K ? D_K1
                                 : (f <= F_AZZ ? D_AT1 + 3 * (f - F_AXX) : D_GAM1 + 3 * (f - F_GAMX)));
            release();
        }
        if (!ok) {   // a wait gave up: report it; the tile's results are dropped
            s_abort = 1;
            atomicExch(a.err, 1);
        }
        if (__any_sync(0xffffffffu, s_abort)) break;
        auto dv = [&](int d) { return my[d * CT]; };
        float hm[4];
        bssn_constraints(u, dv, a.prm, hm);
#pragma unroll
        for (int c = 0; c < 4; c++) cons.c[c][ii] = hm[c];
    }
    // the CTA's shared memory must outlive every copy issued into it: in a normal run all were
    // consumed, after an abort some may be in flight (bounded waits)
    __syncthreads();
    if (tid == 0 && s_abort)
        for (uint32_t n = s_asked, q = n > (uint32_t)R ? n - R : 0u; q < n; q++) mbar_wait(&full[q % R], (q / R) & 1u);
}

// Sum of H^2, max |H|, sum of |M|^2, max |M|^2 and the cell count of a quarter of a listed domain, over its
// interior cells that no child covers and that lie outside the excision radius of every puncture, in double,
// with a fixed order.  Double precision bounds it (two FP64 lanes an SM, so that a square root and the
// maxima in double were two thirds of its time): the maxima compare bits as integers (non-negative numbers
// order alike and a NaN lies above them all), the cells count in integers, and the root is taken once:
// 70 -> 25 us for 264 domains of 16^3.
struct NormSum {
    double h2, m2;
    unsigned long long m_max;   // bits of the largest |M|^2
    uint32_t h_max, cells;      // h_max: bits of the largest |H|
    __device__ __forceinline__ void add(const NormSum& o) {
        h2 += o.h2;
        m2 += o.m2;
        m_max = o.m_max > m_max ? o.m_max : m_max;
        h_max = o.h_max > h_max ? o.h_max : h_max;
        cells += o.cells;
    }
    __device__ __forceinline__ NormSum down(int d) const {
        NormSum o;
        o.h2 = __shfl_down_sync(0xffffffffu, h2, d);
        o.m2 = __shfl_down_sync(0xffffffffu, m2, d);
        o.m_max = __shfl_down_sync(0xffffffffu, m_max, d);
        o.h_max = __shfl_down_sync(0xffffffffu, h_max, d);
        o.cells = __shfl_down_sync(0xffffffffu, cells, d);
        return o;
    }
};
// The CTA's 256 partial sums, added in a fixed order; valid in thread 0.
__device__ __forceinline__ void norm_reduce(NormSum& s) {
    __shared__ NormSum red[8];
#pragma unroll
    for (int d = 16; d > 0; d /= 2) s.add(s.down(d));
    if (threadIdx.x % 32u == 0u) red[threadIdx.x / 32u] = s;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < 8; w++) s.add(red[w]);
}
__global__ void __launch_bounds__(256) k_evo_norms_domain(const __grid_constant__ EvoNormArgs g, double* part) {
    const uint32_t b = blockIdx.x;
    grid_dependency();
    if (b >= g.n_items) return;
    const uint32_t slot = g.items[b], n = g.n, hn = n / 2;
    const uint32_t cells = n * n * n, quarter = cells / kEvoNormParts;
    const uint32_t pos = g.positions[slot];
    const int depth = pos_depth(pos);
    float ctr[3];
    slot_centre(pos, ctr);
    const float h = g.outer_size / ((float)n * (float)(1u << depth));
    NormSum s = {};
    for (uint32_t c = blockIdx.y * quarter + threadIdx.x; c < (blockIdx.y + 1u) * quarter; c += blockDim.x) {
        const uint32_t x = c % n, y = (c / n) % n, z = c / (n * n);
        const uint32_t oct = (x / hn) | ((y / hn) << 1) | ((z / hn) << 2);
        if (g.children[slot * 8u + oct] != -1) continue;
        bool excised = false;
        for (int a = 0; a < g.n_punctures; a++) {
            const float dx = ctr[0] * g.outer_size + ((float)x + .5f - .5f * (float)n) * h - g.pos[a][0];
            const float dy = ctr[1] * g.outer_size + ((float)y + .5f - .5f * (float)n) * h - g.pos[a][1];
            const float dz = ctr[2] * g.outer_size + ((float)z + .5f - .5f * (float)n) * h - g.pos[a][2];
            excised |= dx * dx + dy * dy + dz * dz < g.excision2;
        }
        if (excised) continue;
        const uint64_t i = (uint64_t)slot * cells + c;
        const float hf = g.cons.c[0][i];
        const double hv = hf;
        const double mx = g.cons.c[1][i], my = g.cons.c[2][i], mz = g.cons.c[3][i];
        NormSum e;
        e.h2 = hv * hv;
        e.m2 = mx * mx + my * my + mz * mz;
        e.h_max = __float_as_uint(fabsf(hf));
        e.m_max = (unsigned long long)__double_as_longlong(e.m2);
        e.cells = 1;
        s.add(e);
    }
    norm_reduce(s);
    if (threadIdx.x == 0) {
        double* p = part + ((size_t)b * kEvoNormParts + blockIdx.y) * 5;
        p[0] = s.h2;
        p[1] = __uint_as_float(s.h_max);
        p[2] = s.m2;
        p[3] = __longlong_as_double((long long)s.m_max);
        p[4] = s.cells;
    }
}
// The parts' totals and the norms, in one CTA: thread t adds the parts t, t + 256, ... (a serial sum of
// 264 domains' parts, five loads each, took 107 us).
__global__ void __launch_bounds__(256) k_evo_norms_total(const double* part, uint32_t parts, double* out) {
    grid_dependency();
    NormSum s = {};
    for (uint32_t b = threadIdx.x; b < parts; b += blockDim.x) {
        const double* p = part + (size_t)b * 5;
        NormSum e;
        e.h2 = p[0];
        e.h_max = __float_as_uint((float)p[1]);
        e.m2 = p[2];
        e.m_max = (unsigned long long)__double_as_longlong(p[3]);
        e.cells = (uint32_t)p[4];
        s.add(e);
    }
    norm_reduce(s);
    if (threadIdx.x != 0) return;
    const double cells = s.cells;
    out[0] = s.cells > 0 ? sqrt(s.h2 / cells) : 0.;
    out[1] = __uint_as_float(s.h_max);
    out[2] = s.cells > 0 ? sqrt(s.m2 / cells) : 0.;
    out[3] = sqrt(__longlong_as_double((long long)s.m_max));
    out[4] = cells;
}

template <int N, int TY, int TZ, int R, int MINB>
cudaError_t cons_t(const EvoArgs& a, const ConsPtrs& cons, cudaStream_t st) {
    using S = ConsShape<N, TY, TZ, R, MINB>;
    static std::atomic<uint64_t> configured{0};
    int dev = 0, sms = 0;
    cudaError_t e = ensure_smem_limit(k_evo_constraints<N, TY, TZ, R, MINB>, S::SMEM, configured);
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess || a.n_items == 0) return e;
    const uint32_t tiles = a.n_items * (uint32_t)S::TILES, room = (uint32_t)(sms * MINB);
    k_evo_constraints<N, TY, TZ, R, MINB><<<tiles < room ? tiles : room, S::CT, S::SMEM, st>>>(a, cons);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_evo_constraints(const EvoArgs& a, const ConsPtrs& cons, cudaStream_t st) {
    // the compiled tile depths (evo_deriv_zs_candidates)
    switch (a.n * 16u + a.deriv_zs) {
        case 8 * 16 + 0: case 8 * 16 + 4: return cons_t<8, 8, 4, 4, 2>(a, cons, st);
        case 8 * 16 + 8: return cons_t<8, 8, 8, 8, 1>(a, cons, st);
        case 16 * 16 + 1: return cons_t<16, 16, 1, 3, 2>(a, cons, st);
        case 16 * 16 + 0: case 16 * 16 + 2: return cons_t<16, 16, 2, 6, 1>(a, cons, st);
        case 16 * 16 + 4: return cons_t<16, 8, 4, 6, 1>(a, cons, st);
        case 32 * 16 + 0: case 32 * 16 + 1: return cons_t<32, 16, 1, 4, 1>(a, cons, st);
        default: return cudaErrorInvalidValue;
    }
}
cudaError_t launch_evo_norms(const EvoNormArgs& g, double* part, double* out, cudaStream_t st) {
    if (g.n_items) {
        const cudaError_t e = launch_dependent(true, k_evo_norms_domain, dim3(g.n_items, kEvoNormParts), 256, 0, st, g, part);
        if (e != cudaSuccess) return e;
    }
    return launch_dependent(true, k_evo_norms_total, 1, 256, 0, st, part, g.n_items * kEvoNormParts, out);
}

}  // namespace amr
