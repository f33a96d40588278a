// kernels_evolve.cu -- kernels of the BSSN evolution and of the scalar wave u_tt = Δu (evolve.h).
//
// Compiled with contraction on (-fmad=true): unlike the reference-semantics kernels, these have no
// reference device build to reproduce bit for bit; they are held to the FP64 oracle
// (oracle/bssn_evolve.c) within stated tolerances.
//
//   k_evo_init      analytic initial data on every cell (ghosts included) of every live slot
//   k_evo_stage_wave  one RK4 stage of the wave: derivatives, right-hand side and stage update
//   k_evo_ghost     ghost fill of a stage's state, one face-normal axis per launch (copies from
//                   same-depth neighbours, separable tricubic interpolation from coarser ones)
//   k_evo_restrict  restriction of children into parents, axis by axis (leaves: 16-byte copies)
//   k_evo_prolong   tricubic prolongation of new domains
#include <cmath>
#include <type_traits>

#include "amr_device.cuh"
#include "evolve.h"
#include "evolve_kernels.h"
#include "evolve_physics.cuh"
#include "kernels.h"
#include "tma.cuh"

namespace amr {

namespace {

// ------------------------------------------------------------------ initial data
__global__ void k_evo_init(EvoInitArgs a) {
    const uint32_t t = a.t, cells = t * t * t;
    const uint64_t gid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (uint64_t)a.used * cells) return;
    const uint32_t slot = (uint32_t)(gid / cells), c = (uint32_t)(gid % cells);
    const uint32_t pos = a.positions[slot];
    const int depth = pos_depth(pos);
    if (depth == -1) return;
    float ctr[3];
    slot_centre(pos, ctr);   // exact: sums of powers of two
    const double h = (double)a.outer_size / ((double)a.n * (double)(1u << depth));
    const uint32_t idx[3] = {c % t, (c / t) % t, c / (t * t)};
    double x[3];
    for (int k = 0; k < 3; k++) x[k] = (double)ctr[k] * a.outer_size + ((double)idx[k] + .5 - .5 * (double)t) * h;
    double u[kMaxFields];
    evo_initial_values(a.id, a.physics, x, u);
    for (int f = 0; f < a.nf; f++) {
        const float v = (float)(a.physics == 0 ? u[f] - bssn_offset(f) : u[f]);   // stored as the deviation
        a.out1[f][gid] = v;
        a.out2[f][gid] = v;
        a.out3[f][gid] = v;
    }
}

// ------------------------------------------------------------------ one RK4 stage of the wave
// A CTA per (domain, slab of ZS interior z-planes): the padded planes (ZS + 6) of u and v, one bulk copy
// each, then per cell the Laplacian, the Kreiss-Oliger terms, the right-hand side and the stage update.
// (With a derivative pass and an update kernel, a root step of a root and one child of 16^3 took 62.3 us a pass,
// with this 54.8, most of it launches that depend on one another.)  ZS is a launch-shape choice (amr_sim_autotune times the compiled ones); the default takes
// two cells per thread at 16^3, one at 8^3, four at 32^3.
constexpr int wave_default_zs(int n) { return n == 8 ? 4 : (n == 16 ? 2 : 1); }
template <int N, int ZS>
struct WaveShape {
    static constexpr int T = N + 6, THREADS = 256, CELLS = N * N * ZS, CPT = CELLS / THREADS;
    static constexpr uint32_t SLAB = (uint32_t)((ZS + 6) * T * T);   // floats
    static constexpr size_t SMEM = 2u * SLAB * 4u;
    // The row of a cell.  At N = 16 a warp would cover rows y and y + 1 of the 22-float padded
    // rows, whose shared-memory banks overlap for 6 lanes; rows y and y + 8 (176 floats = 16 banks
    // apart) make every tap of the warp conflict-free.
    __device__ static uint32_t row(uint32_t cell) {
        const uint32_t r = (cell / N) % N;
        return N == 16 ? (r >> 1) | ((r & 1u) << 3) : r;
    }
    static_assert(CELLS % THREADS == 0 && N % ZS == 0, "whole cells per thread and planes per slab");
    static_assert(SLAB * 4u % 16u == 0u && (T * T * 4) % 16 == 0, "slabs are aligned bulk copies");
};

// RK4: stage 1: acc = old + dt/6 k1, out = old + dt/2 k1; stage 2: acc += dt/3 k2, out = old + dt/2 k2;
// stage 3: acc += dt/3 k3, out = old + dt k3; stage 4: out = acc + dt/6 k4.
__device__ __forceinline__ void rk_update(const EvoArgs& a, int f, uint64_t pi, uint64_t ii, float u_old, float r,
                                          float dt) {
    float v;
    switch (a.stage) {
        case 1:
            a.acc[f][ii] = fmaf(dt * (1.f / 6.f), r, u_old);
            v = fmaf(dt * .5f, r, u_old);
            break;
        case 2:
            a.acc[f][ii] = fmaf(dt * (1.f / 3.f), r, a.acc[f][ii]);
            v = fmaf(dt * .5f, r, u_old);
            break;
        case 3:
            a.acc[f][ii] = fmaf(dt * (1.f / 3.f), r, a.acc[f][ii]);
            v = fmaf(dt, r, u_old);
            break;
        default:
            v = fmaf(dt * (1.f / 6.f), r, a.acc[f][ii]);
            break;
    }
    a.out[f][pi] = v;
}

template <int N, int ZS>
__global__ void __launch_bounds__(256) k_evo_stage_wave(const __grid_constant__ EvoArgs a) {
    using S = WaveShape<N, ZS>;
    constexpr int T = S::T;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* buf = reinterpret_cast<float*>(smem_raw);   // u, v
    __shared__ uint64_t bar;
    const uint32_t tid = threadIdx.x;
    grid_dependency();
    const uint32_t item = blockIdx.x / (N / ZS), slab = blockIdx.x % (N / ZS);
    if (item >= a.n_items) return;
    const uint32_t slot = a.items[item];
    if (tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
        mbar_arrive_expect_tx(&bar, 2u * S::SLAB * 4u);
        const size_t src = (size_t)slot * T * T * T + (size_t)slab * ZS * T * T;   // padded plane slab * ZS (p = 3)
        for (int f = 0; f < WAVE_NF; f++) bulk_g2s(buf + (size_t)f * S::SLAB, a.fields[f] + src, S::SLAB * 4u, &bar);
    }
    const int depth = pos_depth(a.positions[slot]);
    const float h = a.prm.outer_size / ((float)N * (float)(1u << depth));
    const float i12h2 = 1.f / (12.f * h * h), ko = a.prm.ko_sigma / (64.f * h);
    const float dt = a.dt0 / (float)(1u << depth);
    __syncthreads();
    const bool ok = mbar_wait(&bar, 0);   // a wait that gave up is reported and its cells are left alone
    if (!ok) atomicExch(a.err, 1);
#pragma unroll
    for (int c = 0; c < S::CPT && ok; c++) {
        const uint32_t cell = tid + (uint32_t)c * S::THREADS;
        const uint32_t x = cell % N, y = S::row(cell), zl = cell / (N * N), z = slab * ZS + zl;
        const uint64_t pi = (uint64_t)slot * T * T * T + ((uint64_t)(z + 3) * T + (y + 3)) * T + (x + 3);
        const uint64_t ii = ((uint64_t)slot * N + z) * N * N + (uint64_t)y * N + x;
        constexpr int st[3] = {1, T, T * T};
        float extra[WAVE_NF], lap = 0.f;
#pragma unroll
        for (int f = 0; f < WAVE_NF; f++) {
            const float* q = buf + (size_t)f * S::SLAB + ((zl + 3) * T + (y + 3)) * T + (x + 3);
            float ko_sum = 0.f, dd[3];
#pragma unroll
            for (int ax = 0; ax < 3; ax++) {
                const int s = st[ax];
                ko_sum += (q[-3 * s] + q[3 * s]) - 6.f * (q[-2 * s] + q[2 * s]) + 15.f * (q[-s] + q[s]) - 20.f * q[0];
                dd[ax] = (16.f * (q[-s] + q[s]) - (q[-2 * s] + q[2 * s]) - 30.f * q[0]) * i12h2;
            }
            if (f == W_U) lap = dd[0] + dd[1] + dd[2];
            extra[f] = __fmul_rn(ko, ko_sum);   // rounded by itself
        }
        const float* q = buf + ((zl + 3) * T + (y + 3)) * T + (x + 3);
        const float uu = q[0], vv = q[S::SLAB];
        const float r_u = vv + extra[W_U], r_v = lap + extra[W_V];
        rk_update(a, W_U, pi, ii, a.stage == 1 ? uu : a.old_f[W_U][pi], r_u, dt);
        rk_update(a, W_V, pi, ii, a.stage == 1 ? vv : a.old_f[W_V][pi], r_v, dt);
    }
    __syncthreads();
    // the CTA's shared memory must outlive its copies: after a wait that gave up, wait once more
    if (!ok && tid == 0) mbar_wait(&bar, 0);
}

// ------------------------------------------------------------------ ghost fill
// Per launch the faces normal to one axis: the host lists those that have a source, the interpolating
// ones (a coarser source) first, as they take longest, then the same-depth copies (evolve_sim.cu).  The
// axis and the domain size are compile-time, so that every division of an index is by a constant.
// Within a launch no cell is both read and written: the fill writes the cells whose index along the axis
// lies in a ghost layer and reads sources inside the interior along it.
//
// Copies: a CTA per (face, kGhostCopyFields fields); a same-depth source is this domain shifted by a whole
// domain, so that rows and planes are moved as 8- and 16-byte vectors (a y face is three whole rows a plane, a z
// face three whole planes; an x face three cells a row), kGhostInFlight loads per thread before their
// stores.
// Interpolations: a CTA per (face, 2 fields), the two fields as the lanes of packed pairs, so that one
// index computation, one shared-memory read and one instruction serve both; the fields of a face in CTAs
// of their own instead of one after another in one CTA, whose twelve synchronised passes were the
// latency of the launch.
// GB300, per launch, before -> now: 585 domains of 16^3, all copies, x 168 -> 124 us (12-byte runs: 1.25
// sectors read and 1.25 written for each, 860 MB of them, 129 us at the copy bandwidth), y 78 -> 54, z 76 -> 47 (326 MB, 49 us);
// nested tree of 201 domains 39 -> 23 on average; two fields beside a coarser domain 13.2 -> 8.3 (latency).
constexpr int kGhostCopyFields = 8, kGhostInFlight = 8;
template <int N, int AXIS>
struct GhostShape {
    static constexpr int P = 3, T = N + 2 * P;
    // extents of the fill: axes before the normal over the whole padded range (their ghosts are
    // filled), axes after it over the interior
    static constexpr int ext(int a) { return a == AXIS ? P : (a < AXIS ? T : N); }
    static constexpr int E0 = ext(0), E1 = ext(1), E2 = ext(2);
    static constexpr int VEC = AXIS == 0 ? 1 : (AXIS == 1 ? 2 : 4);       // floats per copied vector
    static constexpr int COUNT = E0 * E1 * E2 / VEC;                      // vectors per face and field
    static_assert(AXIS != 2 || (T * T) % 4 == 0, "whole planes are 16-byte vectors");
    static_assert(AXIS == 0 || (P * T) % 2 == 0, "whole rows are 8-byte vectors");
    // Interpolation: the largest source box (the source is at least twice as coarse) and the two
    // intermediate stages; the second takes the box's place.
    static constexpr int box(int a) { return ext(a) / 2 + 5; }
    static constexpr int even(int v) { return (v + 1) / 2 * 2; }   // the weights behind them are 16-byte vectors
    static constexpr int BOX = box(0) * box(1) * box(2), ST1 = even(box(2) * box(1) * E0), ST2 = box(2) * E1 * E0;
    static constexpr int FIRST = even(BOX > ST2 ? BOX : ST2);
    static constexpr size_t SMEM = (size_t)(FIRST + ST1) * 8u + (size_t)(E0 + E1 + E2) * 5u * 4u;
};

template <int N, int AXIS>
__global__ void __launch_bounds__(256) k_evo_ghost(const __grid_constant__ EvoGhostArgs g) {
    using S = GhostShape<N, AXIS>;
    constexpr int P = S::P, T = S::T;
    constexpr int64_t CELLS = (int64_t)T * T * T;
    grid_dependency();
    const uint32_t gi = (uint32_t)(g.nf + 1) / 2u, gc = (uint32_t)(g.nf + kGhostCopyFields - 1) / kGhostCopyFields;
    const bool interp = blockIdx.x < g.n_interp * gi;
    const uint32_t b = interp ? blockIdx.x : blockIdx.x - g.n_interp * gi;
    const uint32_t k = interp ? b / gi : g.n_interp + b / gc;
    const uint32_t word = g.faces ? g.faces[k] : g.face[k];   // slot << 1 | side; side 0: + face, 1: - face
    const uint32_t slot = word >> 1, side = word & 1u;
    const uint64_t bd = g.boundaries[(size_t)slot * 6u + AXIS + 3u * side];
    const int32_t src = bd_target(bd);
    const int cd = bd_curr_depth(bd);
    const uint32_t dd = bd_depth_diff(bd);
    const bool src_evolved = g.evolved[src] != 0;
    const float3 relp = cf3_decode((uint32_t)(bd >> 32));
    constexpr int lo_other[3] = {AXIS > 0 ? 0 : P, AXIS > 1 ? 0 : P, P};   // the fill's first index along the other axes
    const int lo_d = side == 0u ? P + N : 0;
    const int lo0 = AXIS == 0 ? lo_d : lo_other[0], lo1 = AXIS == 1 ? lo_d : lo_other[1], lo2 = AXIS == 2 ? lo_d : lo_other[2];

    if (!interp) {   // ---- a same-depth source: active whenever this domain is; its state at the same stage
        const int f0 = (int)(b % gc) * kGhostCopyFields, nfg = min(kGhostCopyFields, g.nf - f0);
        const int r0 = __float2int_rn(relp.x * (float)N), r1 = __float2int_rn(relp.y * (float)N),
                  r2 = __float2int_rn(relp.z * (float)N);
        const int64_t shift = ((int64_t)src - (int64_t)slot) * CELLS + ((int64_t)r2 * T + r1) * T + r0;
        const int64_t dst = (int64_t)slot * CELLS;
        auto move = [&](auto vec, int count, auto cell) {   // count vectors a field, cell(k) their first cell
            using V = decltype(vec);
            const int total = nfg * count;
            for (int e0 = (int)threadIdx.x; e0 < total; e0 += 256 * kGhostInFlight) {
                V v[kGhostInFlight];
#pragma unroll
                for (int i = 0; i < kGhostInFlight; i++) {
                    const int e = e0 + 256 * i;
                    if (e >= total) break;
                    const float* s = src_evolved ? g.X[f0 + e / count] : g.old_f[f0 + e / count];
                    v[i] = *reinterpret_cast<const V*>(s + (dst + shift + cell(e % count)));
                }
#pragma unroll
                for (int i = 0; i < kGhostInFlight; i++) {
                    const int e = e0 + 256 * i;
                    if (e >= total) break;
                    *reinterpret_cast<V*>(g.X[f0 + e / count] + (dst + cell(e % count))) = v[i];
                }
            }
        };
        if constexpr (AXIS == 0) {
            move(0.f, S::COUNT, [&](int q) { return ((q / (P * N) + P) * T + (q / P) % N + P) * T + lo0 + q % P; });
        } else if (shift % S::VEC == 0) {
            if constexpr (AXIS == 1)
                move(float2{}, S::COUNT, [&](int q) { return ((q / (P * T / 2) + P) * T + lo1) * T + 2 * (q % (P * T / 2)); });
            else
                move(float4{}, S::COUNT, [&](int q) { return lo2 * T * T + 4 * q; });
        } else {   // a caller's own boundary record with another offset: cell by cell
            move(0.f, S::COUNT * S::VEC, [&](int q) {
                return ((lo2 + q / (S::E0 * S::E1)) * T + lo1 + (q / S::E0) % S::E1) * T + lo0 + q % S::E0;
            });
        }
        return;
    }
    // ---- A coarser source: separable tricubic interpolation through shared memory.  Along each axis a
    // the ghost cell's coordinate w_a alone gives the base cell b_a of its four-point stencil
    // b_a - 1 .. b_a + 2 and the four Lagrange weights; b_a is kept inside the cells that are
    // valid (the interior along the normal axis and the later axes, the whole padded range along
    // the earlier axes, which earlier passes filled, and everywhere in the root, whose frozen
    // ghost layer is the outer boundary).  b_a grows with w_a, so the source cells read form a
    // box.  The box, with the time interpolation applied to each source cell (frac X + (1 - frac) old, or
    // old alone), then the interpolation along x, along y and along z, each stage through shared memory.
    extern __shared__ __align__(16) unsigned char ghost_smem[];
    float2* const box = reinterpret_cast<float2*>(ghost_smem);   // the source box, then the second stage
    float2* const t1 = box + S::FIRST;                           // [E2][E1][ext0]
    float2* const t2 = box;                                      // [E2][ext1][ext0]
    float* const W = reinterpret_cast<float*>(t1 + S::ST1);      // [ext0 + ext1 + ext2][4] weights
    int* const B = reinterpret_cast<int*>(W + (S::E0 + S::E1 + S::E2) * 4);   // base cells
    const int f0 = (int)(b % gi) * 2, f1 = min(f0 + 1, g.nf - 1);
    const bool root_src = src == 0;
    const bool src_active = active_depth(g.substep, (uint32_t)(cd - (int)dd), g.max_depth);
    // the source's state at the time of the value being filled (evolve.h)
    int mode;      // 0: old only, 2: old..X, 3: old..new
    float frac = 0.f;
    if (!src_evolved) mode = 0;
    else if (src_active) {
        mode = 2;
        frac = 1.f / (float)(1u << dd);
    } else {
        mode = 3;
        const uint32_t kp = (g.substep >> (g.max_depth - (uint32_t)cd)) & ((1u << dd) - 1u);
        frac = ((float)kp + g.c_stage) / (float)(1u << dd);
    }
    const float rel_scale = 1.f / (float)(1u << dd);
    for (int e = (int)threadIdx.x; e < S::E0 + S::E1 + S::E2; e += 256) {
        const int a2 = e < S::E0 ? 0 : (e < S::E0 + S::E1 ? 1 : 2);
        const int j = e - (a2 == 0 ? 0 : (a2 == 1 ? S::E0 : S::E0 + S::E1));
        const int wa = (a2 == 0 ? lo0 : (a2 == 1 ? lo1 : lo2)) + j;
        float rp = ((float)wa - (float)P + .5f) / (float)N - .5f;
        rp = rp * rel_scale + (a2 == 0 ? relp.x : (a2 == 1 ? relp.y : relp.z));
        const float ri = (rp + .5f) * (float)N + (float)P - .5f;
        const int lo_c = root_src || a2 < AXIS ? 1 : P + 1;
        const int hi_c = root_src || a2 < AXIS ? T - 3 : (T - P) - 3;
        int c = __float2int_rd(ri);
        c = c < lo_c ? lo_c : (c > hi_c ? hi_c : c);
        const float x = ri - (float)c;
        B[e] = c;
        float* w = W + e * 4;
        w[0] = -x * (x - 1.f) * (x - 2.f) * (1.f / 6.f);
        w[1] = (x + 1.f) * (x - 1.f) * (x - 2.f) * .5f;
        w[2] = -(x + 1.f) * x * (x - 2.f) * .5f;
        w[3] = (x + 1.f) * x * (x - 1.f) * (1.f / 6.f);
    }
    __syncthreads();
    // the box: from b_min - 1 to b_max + 2 along each axis (the first and the last w_a)
    const int* const B1 = B + S::E0;
    const int* const B2 = B1 + S::E1;
    const int m0 = B[0], m1 = B1[0], m2 = B2[0];
    const int n0 = B[S::E0 - 1] - m0 + 4, n1 = B1[S::E1 - 1] - m1 + 4, n2 = B2[S::E2 - 1] - m2 + 4;
    const int nS = n0 * n1 * n2, nT1 = n2 * n1 * S::E0, nT2 = n2 * S::E1 * S::E0;
    if (nS > S::FIRST || nT1 > S::ST1 || nT2 > S::FIRST) {   // larger than the launch provides: report, skip the face
        if (threadIdx.x == 0) atomicExch(g.err, 1);
        return;
    }
    // e -> (i0, i1, i2) by multiplication: floor(e * ceil(2^21 / n) / 2^21) = floor(e / n) for e < 4332 and
    // n <= 38 (a box has at most 3456 cells)
    const uint32_t q0 = ((1u << 21) + n0 - 1u) / n0, q1 = ((1u << 21) + n1 - 1u) / n1;
    const float* const a00 = g.old_f[f0];
    const float* const a01 = g.old_f[f1];
    const float* const a10 = mode == 3 ? g.new_f[f0] : (const float*)g.X[f0];
    const float* const a11 = mode == 3 ? g.new_f[f1] : (const float*)g.X[f1];
    const int64_t corner = (int64_t)src * CELLS + ((int64_t)(m2 - 1) * T + (m1 - 1)) * T + (m0 - 1);
    const float2 fr = splat2(frac), om = splat2(1.f - frac);
#pragma unroll 4
    for (int e = (int)threadIdx.x; e < nS; e += 256) {
        const uint32_t r = (uint32_t)(((uint64_t)e * q0) >> 21), i2 = (uint32_t)(((uint64_t)r * q1) >> 21);
        const int64_t s = corner + ((int)i2 * T + (int)(r - i2 * n1)) * T + (int)(e - r * n0);
        const float2 o = make_float2(a00[s], a01[s]);
        box[e] = mode == 0 ? o : fma2(fr, make_float2(a10[s], a11[s]), mul2(om, o));
    }
    __syncthreads();
    auto cubic = [&](const float* w, const float2* p, int stride) {
        const float4 c = *reinterpret_cast<const float4*>(w);
        return fma2(splat2(c.w), p[3 * stride], fma2(splat2(c.z), p[2 * stride], fma2(splat2(c.y), p[stride], mul2(splat2(c.x), p[0]))));
    };
    for (int e = (int)threadIdx.x; e < nT1; e += 256) {   // along x
        const int j0 = e % S::E0, r = e / S::E0;          // r = i2 * n1 + i1
        t1[e] = cubic(W + j0 * 4, box + r * n0 + (B[j0] - m0), 1);
    }
    __syncthreads();
    for (int e = (int)threadIdx.x; e < nT2; e += 256) {   // along y
        const int j0 = e % S::E0, r = e / S::E0, j1 = r % S::E1, i2 = r / S::E1;
        t2[e] = cubic(W + (S::E0 + j1) * 4, t1 + (i2 * n1 + (B1[j1] - m1)) * S::E0 + j0, S::E0);
    }
    __syncthreads();
    float* const x0 = g.X[f0] + (int64_t)slot * CELLS;
    float* const x1 = g.X[f1] + (int64_t)slot * CELLS;
    for (int e = (int)threadIdx.x; e < S::E0 * S::E1 * S::E2; e += 256) {   // along z, into the ghost cells
        const int j0 = e % S::E0, r = e / S::E0, j1 = r % S::E1, j2 = r / S::E1;
        const float2 v = cubic(W + (S::E0 + S::E1 + j2) * 4, t2 + ((B2[j2] - m2) * S::E1 + j1) * S::E0 + j0, S::E1 * S::E0);
        const int o = ((lo2 + j2) * T + lo1 + j1) * T + lo0 + j0;
        x0[o] = v.x;
        if (f1 != f0) x1[o] = v.y;
    }
}

// ------------------------------------------------------------------ restriction
// old <- new for every listed slot; a cell covered by a child <- the child's new field at the cell's
// centre (the corner shared by 2x2x2 child cells), by the 4-point midpoint rule (-1, 9, 9, -1)/16 along
// each axis (child cells 2c-1 .. 2c+2, the child's ghost layer at its faces included).  The reference
// averages the 2x2x2 block (AMR.h:961-996), a second-order rule.
//
// One launch, three kinds of CTAs, the longest first: the covered octants' interpolation; the other cells of
// the domains with children, a CTA per (domain, plane, kRestrictCopyFields fields); the domains without,
// straight copies of a plane of every field.
//
// Interpolation: a CTA per (octant, four planes of it, F fields), axis by axis: along x from the child's rows
// (each tap a half of an aligned pair) into shared memory, along y from there into registers, ten planes
// that give four along z.  The sum over 64 taps of every cell was bound by its loads, 64 a cell against 12
// here (20 instructions): 585 domains of 16^3, 73 of them with children, 151 + 306 -> 341 us (the leaves alone 148), 9 of 8^3 5 + 22 -> 5.7.
constexpr int kRestrictCopyFields = 8;
template <int N>
struct RestrictShape {
    static constexpr int T = N + 6, H = N / 2;
    static constexpr int F = N == 8 ? 4 : 256 / (H * H);      // fields per CTA
    static constexpr int SLABS = H / 4, PLANES = 10, ROWS = N + 2;
    static constexpr int PITCH = N == 8 ? 6 : (N == 16 ? 12 : 24);   // floats per row: the y taps of a warp meet no bank twice
    static constexpr int WORDS = F * PLANES * ROWS * PITCH;
    static_assert(F * H * H <= 256 && PITCH >= H && WORDS * 4 <= 48 * 1024, "a column per thread");
};
template <int N>
__global__ void __launch_bounds__(256) k_evo_restrict(const __grid_constant__ EvoRestrictArgs g) {
    using S = RestrictShape<N>;
    constexpr int T = S::T, P = 3, H = S::H;
    constexpr uint64_t CELLS = (uint64_t)T * T * T;
    const uint32_t tid = threadIdx.x;
    grid_dependency();
    uint32_t b = blockIdx.x;
    const uint32_t groups = (uint32_t)(g.nf + S::F - 1) / S::F;
    const uint32_t units = 8u * S::SLABS * groups;      // interpolating CTAs per domain with children
    const uint32_t copies = T * (uint32_t)((g.nf + kRestrictCopyFields - 1) / kRestrictCopyFields);
    if (b < g.n_parents * units) {
        const uint32_t slot = g.items[g.n_leaves + b / units], u = b % units;
        const uint32_t oct = u % 8u, slab = u / 8u % S::SLABS;
        const int f0 = (int)(u / (8u * S::SLABS)) * S::F;
        const int32_t ch = g.children[slot * 8u + oct];
        if (ch == -1) return;
        extern __shared__ float sx[];
        constexpr float wa = -1.f / 16.f, wb = 9.f / 16.f;
        auto four = [](float a, float c, float d, float e) { return fmaf(wa, e, fmaf(wb, d, fmaf(wb, c, wa * a))); };
        // along x: child planes 8 slab - 1 .. 8 slab + 8 and rows -1 .. N of its interior
        const uint64_t src = (uint64_t)ch * CELLS + (uint64_t)(P - 1 + 8 * slab) * T * T + (P - 1) * T + (P - 1);
#pragma unroll 4
        for (int e = (int)tid; e < S::F * S::PLANES * S::ROWS * H; e += 256) {
            const int i = e % H, row = e / H % S::ROWS, z = e / (H * S::ROWS) % S::PLANES, f = e / (H * S::ROWS * S::PLANES);
            if (f0 + f >= g.nf) break;
            const float2* q = reinterpret_cast<const float2*>(g.new_f[f0 + f] + src + (z * T + row) * T + 2 * i);
            const float2 l = q[0], r = q[1];
            sx[((f * S::PLANES + z) * S::ROWS + row) * S::PITCH + i] = four(l.x, l.y, r.x, r.y);
        }
        __syncthreads();
        const int x = (int)tid % H, y = (int)tid / H % H, f = (int)tid / (H * H);
        if (f >= S::F || f0 + f >= g.nf) return;
        float c[S::PLANES];   // along y
#pragma unroll
        for (int z = 0; z < S::PLANES; z++) {
            const float* q = sx + ((f * S::PLANES + z) * S::ROWS + 2 * y) * S::PITCH + x;
            c[z] = four(q[0], q[S::PITCH], q[2 * S::PITCH], q[3 * S::PITCH]);
        }
        float* dst = g.old_f[f0 + f] + slot * CELLS + (uint64_t)(P + (oct >> 2) * H + 4 * slab) * T * T +
                     (P + ((oct >> 1) & 1u) * H + y) * T + P + (oct & 1u) * H + x;
#pragma unroll
        for (int z = 0; z < 4; z++) dst[z * T * T] = four(c[2 * z], c[2 * z + 1], c[2 * z + 2], c[2 * z + 3]);
        return;
    }
    b -= g.n_parents * units;
    if (b < g.n_parents * copies) {
        const uint32_t slot = g.items[g.n_leaves + b / copies], z = b % copies % T;
        const int f0 = (int)(b % copies / T) * kRestrictCopyFields;
        for (int k = (int)tid; k < T * T; k += 256) {
            const uint32_t x = k % T, y = k / T;
            const uint32_t tx = (x - P) / H, ty = (y - P) / H, tz = (z - P) / H;   // unsigned wrap for ghosts
            if (tx < 2u && ty < 2u && tz < 2u && g.children[tx + ty * 2u + tz * 4u + slot * 8u] != -1) continue;
            const uint64_t o = slot * CELLS + (uint64_t)z * T * T + k;
            float v[kRestrictCopyFields];   // every load before the stores (old and new are distinct buffers)
#pragma unroll
            for (int q = 0; q < kRestrictCopyFields; q++)
                if (f0 + q < g.nf) v[q] = g.new_f[f0 + q][o];
#pragma unroll
            for (int q = 0; q < kRestrictCopyFields; q++)
                if (f0 + q < g.nf) g.old_f[f0 + q][o] = v[q];
        }
        return;
    }
    b -= g.n_parents * copies;
    // a plane of every field, 16 bytes at a time (planes are T^2 floats, T^2 * 4 a multiple of 16)
    const uint32_t slot = g.items[b / T], z = b % T;
    constexpr uint32_t q4 = T * T / 4;
    const uint64_t base4 = (slot * CELLS + (uint64_t)z * T * T) / 4u;
    const uint32_t total = (uint32_t)g.nf * q4;
    constexpr uint32_t U = 4;   // loads in flight per thread before their stores
    for (uint32_t e0 = tid; e0 < total; e0 += U * 256u) {
        float4 v[U];
#pragma unroll
        for (uint32_t u = 0; u < U; u++) {
            const uint32_t e = e0 + u * 256u;
            if (e < total) v[u] = reinterpret_cast<const float4*>(g.new_f[e / q4])[base4 + e % q4];
        }
#pragma unroll
        for (uint32_t u = 0; u < U; u++) {
            const uint32_t e = e0 + u * 256u;
            if (e < total) reinterpret_cast<float4*>(g.old_f[e / q4])[base4 + e % q4] = v[u];
        }
    }
}

// ------------------------------------------------------------------ prolongation of new domains
// One CTA per (child, buffer).  Child cell w (padded index) lies at parent index coordinate
// o * n/2 + p + (w - p + 1/2) / 2 - 1/2 along each axis (o: the child's octant bit), which stays in
// [1.25, n + 3.75]: the cubic stencil b-1 .. b+2 (b = floor) fits in the parent's padded range.
// Near a puncture chi ~ r^4 and alpha ~ r^2 (precollapsed lapse): a cubic through their values
// undershoots zero, so they are interpolated as chi^(1/4) and alpha^(1/2), which vary like r, and
// raised back; chi is then kept at or above its floor.
__global__ void __launch_bounds__(256) k_evo_prolong(const __grid_constant__ EvoProlongArgs g) {
    const uint32_t item = blockIdx.x, buf = blockIdx.y;
    if (item >= g.n_items || buf >= g.nbuf) return;
    const int32_t node = g.items[3 * item], parent = g.items[3 * item + 1], off = g.items[3 * item + 2];
    const uint32_t n = g.n, p = g.p, t = g.t;
    const uint64_t cells = (uint64_t)t * t * t;
    const float* src = g.bufs[buf] + (uint64_t)parent * cells;
    float* dst = g.bufs[buf] + (uint64_t)node * cells;
    const uint32_t oct[3] = {(uint32_t)off & 1u, ((uint32_t)off >> 1) & 1u, ((uint32_t)off >> 2) & 1u};
    const float lo = (int)buf == g.floor_buf[0] || (int)buf == g.floor_buf[1] ? g.floor_val : -INFINITY;
    const int root = g.root[buf];
    auto fwd = [&](float v) {   // the interpolated quantity of a stored value
        if (root == 0) return v;
        const float u = sqrtf(fmaxf(v + 1.f, 0.f));
        return root == 2 ? u : sqrtf(u);
    };
    for (uint32_t k = threadIdx.x; k < (uint32_t)cells; k += blockDim.x) {
        const uint32_t w[3] = {k % t, (k / t) % t, k / (t * t)};
        int idx[3];
        float wgt[3][4];
        for (int a = 0; a < 3; a++) {
            const float x = (float)(oct[a] * (n / 2u) + p) + ((float)w[a] - (float)p + .5f) * .5f - .5f;
            int b = __float2int_rd(x);
            b = b < 1 ? 1 : (b > (int)t - 3 ? (int)t - 3 : b);
            const float s = x - (float)b;
            idx[a] = b;
            wgt[a][0] = -s * (s - 1.f) * (s - 2.f) * (1.f / 6.f);
            wgt[a][1] = (s + 1.f) * (s - 1.f) * (s - 2.f) * .5f;
            wgt[a][2] = -(s + 1.f) * s * (s - 2.f) * .5f;
            wgt[a][3] = (s + 1.f) * s * (s - 1.f) * (1.f / 6.f);
        }
        const int64_t si = ((int64_t)idx[2] * t + idx[1]) * t + idx[0];
        float v = 0.f;
#pragma unroll
        for (int k2 = 0; k2 < 4; k2++)
#pragma unroll
            for (int k1 = 0; k1 < 4; k1++) {
                const float w12 = wgt[1][k1] * wgt[2][k2];
                const int64_t row = si + ((int64_t)(k2 - 1) * t + (k1 - 1)) * t - 1;
#pragma unroll
                for (int k0 = 0; k0 < 4; k0++) v = fmaf(wgt[0][k0] * w12, fwd(src[row + k0]), v);
            }
        if (root != 0) {
            const float v2 = v * v;
            v = (root == 2 ? v2 : v2 * v2) - 1.f;
        }
        dst[k] = v < lo ? lo : v;
    }
}

// ------------------------------------------------------------------ tile features and the plain criterion
// One CTA of 512 threads per leaf; thread = cell of the 8^3 feature grid, which covers (N/8)^3
// domain cells.  Per domain cell: the undivided gradients |d chi| and |d alpha| (second-order centred
// differences, i.e. the gradient times the cell size) and |d gt| (the norm over the conformal
// metric's components and axes).  Features of a feature cell: the mean conformal factor,
// log10(max (|d chi| + |d alpha|) + 1e-10) / 5 + 1 and log10(rms |d gt| + 1e-10) / 5 + 1.  The plain
// criterion's indicator of the tile is the largest |d chi| + |d alpha| over its cells.
__global__ void __launch_bounds__(512) k_evo_features(const EvoFeatureArgs g) {
    const uint32_t b = blockIdx.x;
    if (b >= g.n_items) return;
    const uint32_t slot = g.items[b], n = g.n, t = g.t, p = g.p, r = n / 8u;
    const uint32_t c = threadIdx.x, cx = c % 8, cy = (c / 8) % 8, cz = c / 64;
    const uint64_t base = (uint64_t)slot * t * t * t;
    const uint64_t st[3] = {1, t, (uint64_t)t * t};
    float chi = 0.f, g2 = 0.f, ind = 0.f;
    for (uint32_t k = 0; k < r * r * r; k++) {
        const uint32_t x = cx * r + k % r + p, y = cy * r + (k / r) % r + p, z = cz * r + k / (r * r) + p;
        const uint64_t o = base + ((uint64_t)z * t + y) * t + x;
        chi += g.state[F_CHI][o] + bssn_offset(F_CHI);
        float dchi = 0.f, dal = 0.f;
        for (int a = 0; a < 3; a++) {
            const float dc = .5f * (g.state[F_CHI][o + st[a]] - g.state[F_CHI][o - st[a]]);
            const float da = .5f * (g.state[F_ALPHA][o + st[a]] - g.state[F_ALPHA][o - st[a]]);
            dchi += dc * dc;
            dal += da * da;
            for (int q = 0; q < 6; q++) {
                const float dg = .5f * (g.state[F_GXX + q][o + st[a]] - g.state[F_GXX + q][o - st[a]]);
                g2 += dg * dg;
            }
        }
        ind = fmaxf(ind, sqrtf(dchi) + sqrtf(dal));   // per-cell differences are already times dx
    }
    const float inv = 1.f / (float)(r * r * r);
    float* f = g.features + (uint64_t)b * 3u * 512u;
    f[c] = chi * inv;
    f[512 + c] = log10f(ind + 1e-10f) * .2f + 1.f;
    f[1024 + c] = log10f(sqrtf(g2 * inv) + 1e-10f) * .2f + 1.f;
    __shared__ float red[512];
    red[c] = ind;
    __syncthreads();
    for (uint32_t w = 256; w > 0; w >>= 1) {
        if (c < w) red[c] = fmaxf(red[c], red[c + w]);
        __syncthreads();
    }
    if (c == 0) g.indicator[b] = red[0];
}

}  // namespace

// ------------------------------------------------------------------ launchers
cudaError_t launch_evo_prolong(const EvoProlongArgs& g, cudaStream_t st) {
    if (g.n_items == 0 || g.nbuf == 0) return cudaSuccess;
    k_evo_prolong<<<dim3(g.n_items, g.nbuf), 256, 0, st>>>(g);
    return cudaGetLastError();
}

cudaError_t launch_evo_features(const EvoFeatureArgs& g, cudaStream_t st) {
    if (g.n_items == 0) return cudaSuccess;
    k_evo_features<<<g.n_items, 512, 0, st>>>(g);
    return cudaGetLastError();
}

bool evo_config_supported(uint32_t n, uint32_t p) { return p == 3u && (n == 8u || n == 16u || n == 32u); }

cudaError_t launch_evo_init(const EvoInitArgs& a, cudaStream_t st) {
    const uint64_t total = (uint64_t)a.used * a.t * a.t * a.t;
    if (total == 0) return cudaSuccess;
    k_evo_init<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(a);
    return cudaGetLastError();
}

template <int N, int ZS>
static cudaError_t wave_limit() {
    static std::atomic<uint64_t> configured{0};
    return ensure_smem_limit(k_evo_stage_wave<N, ZS>, WaveShape<N, ZS>::SMEM, configured);
}
template <int N, int ZS>
static cudaError_t wave_zs(const EvoArgs& a, cudaStream_t st) {
    using S = WaveShape<N, ZS>;
    const cudaError_t e = wave_limit<N, ZS>();
    if (e != cudaSuccess || a.n_items == 0) return e;
    return launch_dependent(true, k_evo_stage_wave<N, ZS>, a.n_items * (N / ZS), S::THREADS, S::SMEM, st, a);
}
// The compiled slab depths (a.deriv_zs; 0 = the default): whole cells per thread of 256.
template <int N>
static cudaError_t wave_t(const EvoArgs& a, cudaStream_t st) {
    const uint32_t zs = a.deriv_zs ? a.deriv_zs : (uint32_t)wave_default_zs(N);
    if constexpr (N == 8) {
        if (zs == 4) return wave_zs<8, 4>(a, st);
        if (zs == 8) return wave_zs<8, 8>(a, st);
    } else if constexpr (N == 16) {
        if (zs == 1) return wave_zs<16, 1>(a, st);
        if (zs == 2) return wave_zs<16, 2>(a, st);
        if (zs == 4) return wave_zs<16, 4>(a, st);
    } else {
        if (zs == 1) return wave_zs<32, 1>(a, st);
    }
    return cudaErrorInvalidValue;
}
cudaError_t launch_evo_stage_wave(const EvoArgs& a, cudaStream_t st) {
    if (a.n_items != 0 && (a.stage < 1 || a.stage > 4)) return cudaErrorInvalidValue;
    switch (a.n) {
        case 8: return wave_t<8>(a, st);
        case 16: return wave_t<16>(a, st);
        case 32: return wave_t<32>(a, st);
        default: return cudaErrorInvalidValue;
    }
}
uint32_t evo_deriv_zs_candidates(uint32_t n, uint32_t* out) {
    const uint32_t c8[] = {4, 8}, c16[] = {1, 2, 4}, c32[] = {1};
    const uint32_t* c = n == 8 ? c8 : (n == 16 ? c16 : c32);
    const uint32_t k = n == 16 ? 3u : (n == 8 ? 2u : 1u);
    for (uint32_t i = 0; i < k; i++) out[i] = c[i];
    return n == 8 || n == 16 || n == 32 ? k : 0u;
}

template <int N>
static cudaError_t restrict_t(const EvoRestrictArgs& g, cudaStream_t st) {
    using S = RestrictShape<N>;
    const uint32_t units = 8u * S::SLABS * (uint32_t)((g.nf + S::F - 1) / S::F);
    const uint32_t copies = S::T * (uint32_t)((g.nf + kRestrictCopyFields - 1) / kRestrictCopyFields);
    // launches over leaves alone need no shared memory
    return launch_dependent(g.nf == WAVE_NF, k_evo_restrict<N>, g.n_parents * (units + copies) + g.n_leaves * (uint32_t)S::T, 256,
                            g.n_parents ? S::WORDS * 4u : 0u, st, g);
}
cudaError_t launch_evo_restrict(const EvoRestrictArgs& g, cudaStream_t st) {
    if (g.n_leaves + g.n_parents == 0) return cudaSuccess;
    if (g.nf <= 0 || g.nf > kMaxFields) return cudaErrorInvalidValue;
    switch (g.n) {
        case 8: return restrict_t<8>(g, st);
        case 16: return restrict_t<16>(g, st);
        case 32: return restrict_t<32>(g, st);
        default: return cudaErrorInvalidValue;
    }
}

template <int N, int AXIS>
static cudaError_t ghost_limit() {
    static std::atomic<uint64_t> configured{0};
    return ensure_smem_limit(k_evo_ghost<N, AXIS>, GhostShape<N, AXIS>::SMEM, configured);
}
template <int N, int AXIS>
static cudaError_t ghost_t(const EvoGhostArgs& g, cudaStream_t st) {
    const cudaError_t e = ghost_limit<N, AXIS>();
    if (e != cudaSuccess) return e;
    const uint32_t blocks = g.n_interp * (uint32_t)((g.nf + 1) / 2) +
                            g.n_copy * (uint32_t)((g.nf + kGhostCopyFields - 1) / kGhostCopyFields);
    // launches without an interpolating face need none of its shared memory
    return launch_dependent(g.nf == WAVE_NF, k_evo_ghost<N, AXIS>, blocks, 256, g.n_interp ? GhostShape<N, AXIS>::SMEM : 0u, st, g);
}
template <int N>
static cudaError_t ghost_n(const EvoGhostArgs& g, cudaStream_t st) {
    return g.axis == 0 ? ghost_t<N, 0>(g, st) : (g.axis == 1 ? ghost_t<N, 1>(g, st) : ghost_t<N, 2>(g, st));
}
template <int N>
static cudaError_t ghost_limits() {
    cudaError_t e = ghost_limit<N, 0>();
    if (e == cudaSuccess) e = ghost_limit<N, 1>();
    return e == cudaSuccess ? ghost_limit<N, 2>() : e;
}
cudaError_t launch_evo_ghost(const EvoGhostArgs& g, cudaStream_t st) {
    if (g.n_interp + g.n_copy == 0u) return cudaSuccess;
    if (g.axis < 0 || g.axis > 2 || g.nf < 1 || g.nf > kMaxFields) return cudaErrorInvalidValue;
    switch (g.n) {
        case 8: return ghost_n<8>(g, st);
        case 16: return ghost_n<16>(g, st);
        case 32: return ghost_n<32>(g, st);
        default: return cudaErrorInvalidValue;
    }
}
cudaError_t prepare_evo_ghost(uint32_t n) {
    switch (n) {
        case 8: return ghost_limits<8>();
        case 16: return ghost_limits<16>();
        case 32: return ghost_limits<32>();
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace amr
