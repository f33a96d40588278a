// kernels_evolve_stage.cu -- one RK4 stage of the BSSN evolution in a single kernel: derivatives,
// right-hand side and stage update, with every derivative consumed on the SM that computed it.
//
// A derivative pass that writes 93 planes of derivatives and an update that reads them back move
// 93 + 93 values a cell and stage through memory, more than everything else the stage needs (24 fields
// in, 24 out, the step-start values and the accumulator).  Here a persistent CTA takes a tile of one
// domain and visits the 24 fields one after another: each field's padded tile arrives in a ring of
// shared-memory slots by bulk copies, every thread differentiates it at its own cells, and the values
// the algebra needs next wait in a per-thread column of shared memory.  The algebra (Christoffel symbols,
// Ricci tensor, right-hand sides) runs between the groups of visits as soon as a group is complete, so
// that no more than 24 derivatives a cell are ever held.  The stage update's inputs follow through
// the same ring.
//
// A thread takes two cells, z and z + 1, as the lanes of packed f32x2 instructions: a column of eight
// values serves both cells' z differences, and the mixed xz and yz differences share half of their
// taps, 48 shared-memory loads a cell and field instead of 67.  The loops over a group's fields are
// not unrolled: the unrolled kernel (80 KB of code) spent 41 % of its time waiting for instructions and
// ran at 856 us a launch against 470.
//
// The values of the first and last three layers of cells along an axis are also written to the ghost layers of
// the same-depth neighbours that copy them (EvoArgs::feed), edges and corners by way of two or three of them.
// A fill of those layers by itself reads what was just written, along x in 12-byte runs: x 124, y 54 and z 47 us
// a stage of the uniform depth-3 tree (evo_stage_feeds has the rule and a root step's times).
//
// Measured on a GB300, 585 domains of 16^3 (2.40 M cells), one stage: 779 us for the two kernels it
// replaces (317 + 462 on average over the stages), 470 us by itself and 545 with x and y fed; a root step of the
// uniform depth-3 tree 38.4 -> 28.2 ms with this kernel alone, 20.1 now with the fed ghosts and the other
// kernels' changes.  What bounds it: the latency of eight warps (38 % of the issue slots, 54 % of the shared-memory pipe, about 1 180
// wavefronts per 32 cells) in the visits and, in the update, the memory traffic that all SMs issue at the
// same time; the two do not overlap, as a CTA's registers and columns fill its SM.  One cell a thread and
// twice the warps gave 30.0 ms; the update spread over the next tile's visits was 3 % faster with warm
// caches and 3 to 5 % slower on small trees with cold ones.
//
// Compiled with contraction on, as kernels_evolve.cu (held to the FP64 oracle, no reference build to
// reproduce).
#include <type_traits>

#include "amr_device.cuh"
#include "evolve.h"
#include "evolve_kernels.h"
#include "kernels.h"
#include "tma.cuh"

namespace amr {

namespace {

// A thread's cells: one, or z and z + 1 as the lanes of packed pairs.
struct V1 {
    float v;
    static constexpr int L = 1;
    static __device__ __forceinline__ V1 splat(float x) { return V1{x}; }
    static __device__ __forceinline__ V1 ld(const float* q, int) { return V1{q[0]}; }   // q[i * stride] per cell i
    __device__ __forceinline__ void st(float* q, int, uint32_t cells = 1u) const { if (cells & 1u) q[0] = v; }
};
struct V2 {
    float2 v;
    static constexpr int L = 2;
    static __device__ __forceinline__ V2 splat(float x) { return V2{make_float2(x, x)}; }
    static __device__ __forceinline__ V2 ld(const float* q, int stride) { return V2{make_float2(q[0], q[stride])}; }
    __device__ __forceinline__ void st(float* q, int stride, uint32_t cells = 3u) const {   // bit i: cell i
        if (cells & 1u) q[0] = v.x;
        if (cells & 2u) q[stride] = v.y;
    }
};
__device__ __forceinline__ V2 mk(float x, float y) { return V2{make_float2(x, y)}; }
__device__ __forceinline__ V2 operator+(V2 a, V2 b) { return V2{__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ V2 operator*(V2 a, V2 b) { return V2{__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ V2 operator-(V2 a, V2 b) { return V2{__ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v)}; }
__device__ __forceinline__ V2 fma(V2 a, V2 b, V2 c) { return V2{__ffma2_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ V2 fma(float a, V2 b, V2 c) { return fma(V2::splat(a), b, c); }
__device__ __forceinline__ V2 operator*(float s, V2 a) { return V2::splat(s) * a; }
__device__ __forceinline__ V1 operator+(V1 a, V1 b) { return V1{a.v + b.v}; }
__device__ __forceinline__ V1 operator*(V1 a, V1 b) { return V1{a.v * b.v}; }
__device__ __forceinline__ V1 operator-(V1 a, V1 b) { return V1{a.v - b.v}; }
__device__ __forceinline__ V1 fma(V1 a, V1 b, V1 c) { return V1{fmaf(a.v, b.v, c.v)}; }
__device__ __forceinline__ V1 fma(float a, V1 b, V1 c) { return V1{fmaf(a, b.v, c.v)}; }
__device__ __forceinline__ V1 operator*(float s, V1 a) { return V1{s * a.v}; }
__device__ __forceinline__ V2 recip(V2 a) { return mk(1.f / a.v.x, 1.f / a.v.y); }
__device__ __forceinline__ V1 recip(V1 a) { return V1{1.f / a.v}; }
// max(a, lo), keeping a NaN (at_least) or replacing it (floor_at)
__device__ __forceinline__ V2 at_least(V2 a, float lo) { return mk(a.v.x < lo ? lo : a.v.x, a.v.y < lo ? lo : a.v.y); }
__device__ __forceinline__ V1 at_least(V1 a, float lo) { return V1{a.v < lo ? lo : a.v}; }
__device__ __forceinline__ V2 floor_at(V2 a, float lo) { return mk(fmaxf(a.v.x, lo), fmaxf(a.v.y, lo)); }
__device__ __forceinline__ V1 floor_at(V1 a, float lo) { return V1{fmaxf(a.v, lo)}; }

// The visiting order of the fields of a tile: the metric first (its inverse contracts the second
// derivatives), then each group when its derivatives can be consumed, the shift last.
constexpr int kVisits = BSSN_NF;
__device__ __forceinline__ int stage_field(int i, bool shift_on) {
    if (i < 6) return F_GXX + i;
    if (i < 8) return i == 6 ? F_CHI : F_ALPHA;
    if (i < 12) return i == 11 ? F_K : F_GAMX + (i - 8);
    if (i < 18) return F_AXX + (i - 12);
    return shift_on && i < 21 ? F_BX + (i - 18) : F_BETAX + (i - (shift_on ? 21 : 18));
}
// Per-thread values in shared memory: the extra terms of the 24 fields, the outputs of the current
// group of visits (24, and at the end the right-hand sides), and values parked between groups.
constexpr int P_T = BSSN_NF, P_X = P_T + 6 /* while the group's outputs are the curvature's six */, P_GAM = P_T + 24,
              P_GC = P_GAM + 3, P_B = P_GC + 3, kStash = P_B + 3;

// A tile of N x TY x TZ interior cells of one domain; a field's padded tile (TY + 6 rows of TZ + 6
// planes, each plane's rows contiguous in the field) is one ring slot, a bulk copy per plane.
template <int N, int TY, int TZ, int R_, int L>
struct StageShape {
    static constexpr int T = N + 6;
    static constexpr int CT = N * TY * TZ / L;            // threads, L cells each
    static constexpr int WARPS = CT / 32;
    static constexpr int ROWS = TY + 6, PLANES = TZ + 6;
    static constexpr int CHUNK = ROWS * T;                // floats per plane
    static constexpr bool WHOLE = TY == N;                // whole planes: a field's tile is one copy
    // plane pitch of a tile of part planes: the half warps of 16^3 domains take cells L planes
    // apart, whose banks must lie 16 apart: L * PP = 16 mod 32
    static constexpr int pitch() {
        int p = CHUNK;
        if (!WHOLE && N == 16) while ((L * p) % 32 != 16) p += 4;
        return p;
    }
    static constexpr int PP = pitch();
    static constexpr int SLOT = PLANES * PP;              // floats
    // The stage update's inputs come through the ring too, F fields per slot: the step-start values
    // (rows from y0 + 2 to y0 + TY + 3, which makes the copies 16-byte aligned) and the accumulator.
    static constexpr int OLD_PLANE = WHOLE ? T * T : (TY + 2) * T;                   // floats from z to z + 1
    static constexpr int OLD_F = (TZ - 1) * OLD_PLANE + (TY + 2) * T, ACC_F = TZ * TY * N;
    static constexpr int fields_per_slot() {
        for (int f : {4, 3, 2})
            if (f * (OLD_F + ACC_F) <= SLOT) return f;
        return 1;
    }
    static constexpr int F = fields_per_slot(), UPDATES = BSSN_NF / F;
    // ring slots, and how many visits ahead a field is requested: two less than the slots, so that
    // the slot to be refilled was released two visits ago by all but the slowest warps
    static constexpr int R = R_, AHEAD = R - 2;
    static constexpr int TILES = (N / TY) * (N / TZ);
    static constexpr size_t SMEM = ((size_t)R * SLOT + (size_t)kStash * CT * L) * 4u + 2u * R * 8u;
    static_assert(CT % 32 == 0 && TZ % L == 0 && N % TY == 0 && N % TZ == 0, "whole warps of cell pairs");
    static_assert((CHUNK * 4) % 16 == 0 && (TY * T * 4) % 16 == 0 && (T * T * 4) % 16 == 0 && PP % 4 == 0 && PLANES <= 32,
                  "every plane is an aligned bulk copy");
    static_assert(OLD_F + ACC_F <= SLOT && OLD_F % 4 == 0 && OLD_PLANE % 4 == 0 && ACC_F % 4 == 0 && (2 * T * 4) % 16 == 0 &&
                  (!WHOLE || PP == T * T) && (TY * N * 4) % 16 == 0, "the update's inputs are aligned bulk copies");
    static_assert(SMEM <= 227u * 1024u, "fits an SM");
};

__device__ __forceinline__ int si(int i, int j) {        // xx xy xz yy yz zz
    const int a = i < j ? i : j, b = i < j ? j : i;
    return a == 0 ? b : (a == 1 ? 2 + b : 5);
}

// Unscaled derivatives of one field at a thread's two cells, from its tile: D = 12 h d_a, S = -12 h^2
// d_a d_a, M = 144 h^2 d_a d_b (xy, xz, yz), and the field's extra term: advection along the shift
// (b = shift / 12 h) plus Kreiss-Oliger dissipation (ko = sigma / 64 h).
template <class V>
struct Der {
    V q, D[3], S[3], M[3], extra;
};
template <int T, int PP, bool SECOND, class V>
__device__ __forceinline__ void derive(const float* q, const V* b, float ko, Der<V>& o) {
    auto pr = [&](int k) { return V::ld(q + k, PP); };
    V z1, z1n, z2, z2n, z3, z3n;
    if constexpr (V::L == 2) {   // eight consecutive planes give the seven pairs along z
        float zc[8];
#pragma unroll
        for (int k = 0; k < 8; k++) zc[k] = q[(k - 3) * PP];
        o.q = mk(zc[3], zc[4]);
        z1 = mk(zc[4], zc[5]); z1n = mk(zc[2], zc[3]);
        z2 = mk(zc[5], zc[6]); z2n = mk(zc[1], zc[2]);
        z3 = mk(zc[6], zc[7]); z3n = mk(zc[0], zc[1]);
    } else {
        o.q = pr(0);
        z1 = pr(PP); z1n = pr(-PP); z2 = pr(2 * PP); z2n = pr(-2 * PP); z3 = pr(3 * PP); z3n = pr(-3 * PP);
    }
    const V x1 = pr(1), x1n = pr(-1), x2 = pr(2), x2n = pr(-2);
    const V y1 = pr(T), y1n = pr(-T), y2 = pr(2 * T), y2n = pr(-2 * T);
    o.D[0] = fma(8.f, x1 - x1n, x2n - x2);
    o.D[1] = fma(8.f, y1 - y1n, y2n - y2);
    o.D[2] = fma(8.f, z1 - z1n, z2n - z2);
    const V sx1 = x1 + x1n, sy1 = y1 + y1n, sz1 = z1 + z1n;
    const V sx2 = x2 + x2n, sy2 = y2 + y2n, sz2 = z2 + z2n;
    const V s3 = (pr(3) + pr(-3)) + (pr(3 * T) + pr(-3 * T)) + (z3 + z3n);
    const V s1 = sx1 + sy1 + sz1, s2 = sx2 + sy2 + sz2;
    const V dis = fma(-60.f, o.q, fma(15.f, s1, fma(-6.f, s2, s3)));
    o.extra = fma(b[0], o.D[0], fma(b[1], o.D[1], fma(b[2], o.D[2], ko * dis)));
    if constexpr (SECOND) {
        // the large terms meet in one rounding, as late as possible
        o.S[0] = fma(30.f, o.q, fma(-16.f, sx1, sx2));
        o.S[1] = fma(30.f, o.q, fma(-16.f, sy1, sy2));
        o.S[2] = fma(30.f, o.q, fma(-16.f, sz1, sz2));
        auto dx = [&](int k) { return fma(8.f, pr(k + 1) - pr(k - 1), pr(k - 2) - pr(k + 2)); };
        auto dy = [&](int k) { return fma(8.f, pr(k + T) - pr(k - T), pr(k - 2 * T) - pr(k + 2 * T)); };
        o.M[0] = fma(8.f, dx(T) - dx(-T), dx(-2 * T) - dx(2 * T));
        if constexpr (V::L == 2) {   // planes z - 2, z - 1 and z + 2, z + 3; z and z + 1 are the first derivatives
            const V lx = dx(-2 * PP), hx = dx(2 * PP);
            o.M[1] = fma(8.f, mk(o.D[0].v.y, hx.v.x) - mk(lx.v.y, o.D[0].v.x), lx - hx);
            const V ly = dy(-2 * PP), hy = dy(2 * PP);
            o.M[2] = fma(8.f, mk(o.D[1].v.y, hy.v.x) - mk(ly.v.y, o.D[1].v.x), ly - hy);
        } else {
            o.M[1] = fma(8.f, dx(PP) - dx(-PP), dx(-2 * PP) - dx(2 * PP));
            o.M[2] = fma(8.f, dy(PP) - dy(-PP), dy(-2 * PP) - dy(2 * PP));
        }
    }
}

// gt^ij m_ij of a symmetric m, with g the inverse metric (xx xy xz yy yz zz)
template <class V>
__device__ __forceinline__ V trace(const V* g, const V* m) {
    const V d = fma(g[0], m[0], fma(g[3], m[3], g[5] * m[5]));
    const V o = fma(g[1], m[1], fma(g[2], m[2], g[4] * m[4]));
    return fma(2.f, o, d);
}

template <int N, int TY, int TZ, int R_, class V, int MINB, int FEED>
__global__ void __launch_bounds__(StageShape<N, TY, TZ, R_, V::L>::CT, MINB)
    k_evo_stage_bssn(const __grid_constant__ EvoArgs a) {
    using S = StageShape<N, TY, TZ, R_, V::L>;
    constexpr int T = S::T, PP = S::PP, R = S::R, CT = S::CT, L = V::L;
    auto sp = [](float v) { return V::splat(v); };
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* ring = reinterpret_cast<float*>(smem_raw);
    V* stash = reinterpret_cast<V*>(ring + (size_t)R * S::SLOT);   // [value][thread]
    uint64_t* full = reinterpret_cast<uint64_t*>(stash + (size_t)kStash * CT);
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
    __syncthreads();
    const uint32_t tiles = a.n_items * (uint32_t)S::TILES;
    const bool shift_on = a.prm.shift != 0;
    const int visits = shift_on ? kVisits : kVisits - 3;   // a frozen shift's driver is not differentiated
    const int all_visits = visits + S::UPDATES;
    bool ok = true;
    const uint32_t spins = a.spin_limit ? a.spin_limit : kMaxSpins;

    // Request visit i of tile t (of domain `slot`), the q-th of this CTA, by one whole warp, once every
    // warp has released the slot's previous contents.  Visits 0 .. visits - 1 bring a field's tile
    // each, the others the stage update's inputs.  Whole planes are one copy, part planes one a plane.
    const bool use_old = a.stage != 4, use_acc = a.stage != 1;
    auto request = [&](uint32_t q, uint32_t t, uint32_t slot, int i) {
        if (t >= tiles) return;
        const uint32_t s = q % R;
        // the whole warp or none of it: no lane's copy is issued without lane 0's announcement, as nothing would
        // wait for it
        ok = __all_sync(0xffffffffu, ok && (q < (uint32_t)R || mbar_wait(&empty[s], ((q / R) - 1u) & 1u, spins)));
        if (!ok) return;
        const uint32_t k = t % S::TILES, z0 = (k / (N / TY)) * TZ, y0 = (k % (N / TY)) * TY;
        float* dst = ring + (size_t)s * S::SLOT;
        const bool tile = i < visits;
        if (lane == 0) {
            const uint32_t held = q + 1u == a.withhold;   // failure-path test: more announced than comes
            mbar_arrive_expect_tx(&full[s], 4u * (tile ? (uint32_t)(S::PLANES * S::CHUNK)
                                                   : (uint32_t)S::F * ((use_old ? (S::WHOLE ? S::OLD_F : TZ * (TY + 2) * T) : 0) +
                                                                       (use_acc ? S::ACC_F : 0))) + held);
            atomicMax(&s_asked, q + 1u);   // the warps' requests may pass one another
        }
        __syncwarp();
        const size_t plane = (size_t)slot * T + z0;   // the first padded plane
        if (tile) {
            const float* src = a.fields[stage_field(i, shift_on)] + plane * T * T + (size_t)y0 * T;
            if constexpr (S::WHOLE) {
                if (lane == 0) bulk_g2s(dst, src, S::SLOT * 4u, &full[s]);
            } else {
                if (lane < (uint32_t)S::PLANES) bulk_g2s(dst + (size_t)lane * PP, src + (size_t)lane * T * T, S::CHUNK * 4u, &full[s]);
            }
        } else {
            const int f0 = (i - visits) * S::F;
#pragma unroll 1
            for (int j = 0; j < S::F; j++, dst += S::OLD_F + S::ACC_F) {
                const float* o = a.old_f[f0 + j] + (plane + 3u) * T * T + (size_t)(y0 + 2u) * T;
                const float* c = a.acc[f0 + j] + ((size_t)slot * N + z0) * N * N + (size_t)y0 * N;
                if constexpr (S::WHOLE) {
                    if (lane == 0 && use_old) bulk_g2s(dst, o, S::OLD_F * 4u, &full[s]);
                    if (lane == 0 && use_acc) bulk_g2s(dst + S::OLD_F, c, S::ACC_F * 4u, &full[s]);
                } else if (lane < (uint32_t)TZ) {
                    if (use_old) bulk_g2s(dst + (size_t)lane * S::OLD_PLANE, o + (size_t)lane * T * T, (TY + 2) * T * 4u, &full[s]);
                    if (use_acc) bulk_g2s(dst + S::OLD_F + (size_t)lane * TY * N, c + (size_t)lane * N * N, TY * N * 4u, &full[s]);
                }
            }
        }
    };
    uint32_t nslot = a.items[blockIdx.x / S::TILES];   // the next tile's slot
    if (warp == 0)
        for (int i = 0; i < S::AHEAD; i++) request(i, blockIdx.x, nslot, i);   // AHEAD <= visits

    // thread (x, z of the first cell, y): at N = 16 the half warps take rows 8 apart (176 floats = 16
    // banks) of whole planes, or z-pairs 2 planes apart of part planes
    const uint32_t x = tid % N;
    uint32_t r = tid / N, zl, y;
    if constexpr (S::WHOLE && N == 16) {
        y = ((r >> 1) & 7u) | ((r & 1u) << 3);
        zl = (r >> 4) * L;
    } else if constexpr (S::WHOLE && N == 8 && TZ == 8 && L == 1) {   // quarter warps 2 planes (392 floats = 8 banks) apart
        zl = 2u * (r & 3u) + ((r >> 2) & 1u);
        y = r >> 3;
    } else {
        zl = (r % (TZ / L)) * L;
        y = r / (TZ / L);
    }
    const int c0 = (int)(zl + 3) * PP + (int)(y + 3) * T + (int)x + 3;
    V* const my = stash + tid;
    uint32_t v = 0;   // visits consumed
    // the metric and the shift at this thread's cells of tile t, loaded before its visits
    V own[9];
    // the tile's padded and inner index of cell z (z + 1 lies a plane on); 32 bits are enough, as the 72
    // padded buffers of a simulation fit the device's memory
    uint32_t npi = 0, nii = 0;
    // Feeding: the side of the domain (0: its first layers, 1: its last, -1: neither) along an axis of this
    // thread's cells, and the domains fed along each axis (-1: none), asked for with the tile's metric
    auto side = [](uint32_t w) { return w < 3u ? 0 : (w >= N - 3u ? 1 : -1); };
    auto side_z = [&](uint32_t z) { return L == 2 && side(z) < 0 ? side(z + 1u) : side(z); };
    auto next_domain = [&](int32_t in, int axis, int s) { return in >= 0 && s >= 0 ? a.feed[6 * in + 2 * axis + s] : -1; };
    const int sx = side(x);
    int32_t ndx = -1, ndy = -1, ndz = -1;
    int ndepth = 0;
    auto load_own = [&](uint32_t t) {   // of tile t, in domain nslot
        const uint32_t k = t % S::TILES, z = (k / (N / TY)) * TZ + zl, yy = (k % (N / TY)) * TY + y;
        npi = (nslot * T + z + 3) * T * T + (yy + 3) * T + x + 3;
        nii = (nslot * N + z) * N * N + yy * N + x;
        ndepth = pos_depth(a.positions[nslot]);
        if (FEED > 0 && a.feed) {
            ndx = next_domain((int32_t)nslot, 0, sx);
            if (FEED > 1) ndy = next_domain((int32_t)nslot, 1, side(yy));
            if (FEED > 2) ndz = next_domain((int32_t)nslot, 2, side_z(z));
        }
#pragma unroll
        for (int i = 0; i < 9; i++) {
            const float* q = a.fields[i < 6 ? F_GXX + i : F_BETAX + (i - 6)] + npi;
            own[i] = V::ld(q, T * T);
        }
    };
    load_own(blockIdx.x);   // the grid has no more CTAs than tiles
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t pi = npi, ii = nii, slot = nslot;
        const int depth = ndepth;
        // the domains at the edges and the corner, by way of the neighbours along the earlier axes
        const uint32_t tk = t % S::TILES, cz = (tk / (N / TY)) * TZ + zl;
        const int sy = side((tk % (N / TY)) * TY + y), sz = side_z(cz);
        uint32_t zmask = 0u;   // bit i: cell i lies in the side's layers along z
#pragma unroll
        for (int i = 0; i < L; i++) zmask |= FEED > 2 && side(cz + i) >= 0 ? 1u << i : 0u;
        const int32_t dx = ndx, dy = ndy, dz = ndz;
        const int32_t dxy = FEED > 1 ? next_domain(dx, 1, sy) : -1;
        const int32_t dxz = FEED > 2 ? next_domain(dx, 2, sz) : -1, dyz = FEED > 2 ? next_domain(dy, 2, sz) : -1;
        if (t + gridDim.x < tiles) nslot = a.items[(t + gridDim.x) / S::TILES];
        const float h = a.prm.outer_size / ((float)N * (float)(1u << depth));
        const float i12h = 1.f / (12.f * h), i12h2 = 1.f / (12.f * h * h), i144h2 = 1.f / (144.f * h * h);
        const float ko = a.prm.ko_sigma / (64.f * h);
        V b[3], g[6];
#pragma unroll
        for (int i = 0; i < 3; i++) b[i] = i12h * own[6 + i];
#pragma unroll
        for (int i = 0; i < 6; i++) g[i] = own[i] + sp(i == 0 || i == 3 || i == 5 ? 1.f : 0.f);
        // The tile's next field: the warps take turns to request the field AHEAD visits on, then wait.
        int vi = 0;   // visits of this tile
        auto wait = [&](uint32_t p) { ok = mbar_wait(&full[p % R], (p / R) & 1u, spins) && ok; };
        auto visit = [&]() {
            if (warp == (uint32_t)vi % S::WARPS) {
                const int j = vi + S::AHEAD;
                if (j < all_visits) request(v + S::AHEAD, t, slot, j);
                else request(v + S::AHEAD, t + gridDim.x, nslot, j - all_visits);
            }
            vi++;
            wait(v);
        };
        auto tile = [&](uint32_t p) { return ring + (size_t)(p % R) * S::SLOT + c0; };
        auto release = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[v % R]);
            v++;
        };
        auto keep = [&](int f, V e) { my[(size_t)f * CT] = e; };
        auto back = [&](int f) { return my[(size_t)f * CT]; };
        // ---- the metric: values, inverse, derivatives
        V gi[6];
        {
            const V c00 = g[3] * g[5] - g[4] * g[4], c01 = g[2] * g[4] - g[1] * g[5], c02 = g[1] * g[4] - g[2] * g[3];
            const V id = recip(fma(g[0], c00, fma(g[1], c01, g[2] * c02)));
            gi[0] = c00 * id;
            gi[1] = c01 * id;
            gi[2] = c02 * id;
            gi[3] = (g[0] * g[5] - g[2] * g[2]) * id;
            gi[4] = (g[1] * g[2] - g[0] * g[4]) * id;
            gi[5] = (g[0] * g[3] - g[1] * g[1]) * id;
        }
        // gt^lm d_l d_m of a field, from its unscaled second derivatives
        auto lap = [&](const Der<V>& d) {
            const V s = fma(gi[0], d.S[0], fma(gi[3], d.S[1], gi[5] * d.S[2]));
            const V m = fma(gi[1], d.M[0], fma(gi[2], d.M[1], gi[4] * d.M[2]));
            return fma(-i12h2, s, (2.f * i144h2) * m);
        };
#pragma unroll 1
        for (int c = 0; c < 6; c++) {
            visit();
            Der<V> d;
            derive<T, PP, true>(tile(v), b, ko, d);
            release();
            keep(F_GXX + c, d.extra);
#pragma unroll
            for (int j = 0; j < 3; j++) keep(P_T + 3 * c + j, d.D[j]);   // 12 h d_j gt_c
            keep(P_T + 18 + c, lap(d));
        }
        // lowered Christoffel symbols Gt_ijk = (d_j gt_ik + d_k gt_ij - d_i gt_jk) / 2, and raised
        V cu[3][6], Rc[6];   // Gt^i_jk; the Ricci tensor
        {
            V cl[3][6];
            const float hs = .5f * i12h;
            auto dg = [&](int c, int j) { return back(P_T + 3 * c + j); };
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++)
#pragma unroll
                    for (int l = j; l < 3; l++) {
                        V w;
                        if (i == j) w = hs * dg(si(i, i), l);           // d_l gt_ii / 2
                        else if (i == l) w = hs * dg(si(i, i), j);
                        else if (j == l) w = fma(i12h, dg(si(i, j), j), (-hs) * dg(si(j, j), i));
                        else w = hs * ((dg(si(i, l), j) + dg(si(i, j), l)) - dg(si(j, l), i));
                        cl[i][si(j, l)] = w;
                    }
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int c = 0; c < 6; c++)
                    cu[i][c] = fma(gi[si(i, 0)], cl[0][c], fma(gi[si(i, 1)], cl[1][c], gi[si(i, 2)] * cl[2][c]));
            // Gt_d^k Gt_(ij)k
            V gd[3];
#pragma unroll
            for (int i = 0; i < 3; i++) gd[i] = .5f * trace(gi, cu[i]);
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = i; j < 3; j++)
#pragma unroll
                    for (int l = 0; l < 3; l++) {
                        const V w = cl[i][si(j, l)] + cl[j][si(i, l)];
                        Rc[si(i, j)] = l == 0 ? gd[l] * w : fma(gd[l], w, Rc[si(i, j)]);
                    }
            // gt^lm (Gt^k_li Gt_jkm + Gt^k_lj Gt_ikm + Gt^k_im Gt_klj): with Q_i^km = gt^ml Gt^k_li the
            // three terms are Q_i^km Gt_jkm, Q_j^km Gt_ikm and Q_i^km Gt_kmj
#pragma unroll
            for (int i = 0; i < 3; i++) {
                V Q[3][3];
#pragma unroll
                for (int l = 0; l < 3; l++)
#pragma unroll
                    for (int m = 0; m < 3; m++)
                        Q[l][m] = fma(gi[si(m, 0)], cu[l][si(0, i)], fma(gi[si(m, 1)], cu[l][si(1, i)], gi[si(m, 2)] * cu[l][si(2, i)]));
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    V s = Q[0][0] * cl[j][si(0, 0)];
#pragma unroll
                    for (int l = 0; l < 3; l++)
#pragma unroll
                        for (int m = 0; m < 3; m++)
                            if (l || m) s = fma(Q[l][m], cl[j][si(l, m)], s);
                    V r = fma(i == j ? 2.f : 1.f, s, Rc[si(i, j)]);
                    if (j >= i) {
#pragma unroll
                        for (int l = 0; l < 3; l++)
#pragma unroll
                            for (int m = 0; m < 3; m++) r = fma(Q[l][m], cl[l][si(m, j)], r);
                    }
                    Rc[si(i, j)] = r;
                }
            }
            // The second derivatives' part last: the terms above are small beside it, and would each be rounded at
            // its size.  (With it first, and the connection functions' products added one by one, the errors against
            // 64 bits were 0.8 % above those of the two kernels before after one step of 9 domains of 8^3, 0.1 %
            // after eight; now 0.5 % above and 0.04 % below, means over 24 states and 18 fields.)
#pragma unroll
            for (int c = 0; c < 6; c++) Rc[c] = fma(-.5f, back(P_T + 18 + c), Rc[c]);
        }
        const int32_t dxyz = FEED > 2 ? next_domain(dxy, 2, sz) : -1;
        // ---- the conformal factor and the lapse
#pragma unroll 1
        for (int l = 0; l < 2; l++) {
            visit();
            Der<V> d;
            derive<T, PP, true>(tile(v), b, ko, d);
            release();
            keep(l == 0 ? F_CHI : F_ALPHA, d.extra);
            keep(P_T + 10 * l, d.q);
#pragma unroll
            for (int j = 0; j < 3; j++) {
                keep(P_T + 10 * l + 1 + j, i12h * d.D[j]);
                keep(P_T + 10 * l + 4 + 3 * (j == 1) + 5 * (j == 2), -i12h2 * d.S[j]);   // xx yy zz
            }
            keep(P_T + 10 * l + 5, i144h2 * d.M[0]);
            keep(P_T + 10 * l + 6, i144h2 * d.M[1]);
            keep(P_T + 10 * l + 8, i144h2 * d.M[2]);
        }
        V chi, alpha, nlap, p[3], dal[3];   // p = d chi / (2 max(chi, floor)); nlap = -D^i D_i alpha
        {
            chi = back(P_T) + sp(1.f);
            alpha = back(P_T + 10) + sp(1.f);
            const V hi2 = .5f * recip(floor_at(chi, a.prm.chi_floor));
            V dc[3], w[3], dd[6];
#pragma unroll
            for (int i = 0; i < 3; i++) { dc[i] = back(P_T + 1 + i); dal[i] = back(P_T + 11 + i); p[i] = hi2 * dc[i]; }
#pragma unroll
            for (int c = 0; c < 6; c++)
                dd[c] = back(P_T + 4 + c) - fma(cu[0][c], dc[0], fma(cu[1][c], dc[1], cu[2][c] * dc[2]));
#pragma unroll
            for (int i = 0; i < 3; i++) w[i] = fma(gi[si(i, 0)], dc[0], fma(gi[si(i, 1)], dc[1], gi[si(i, 2)] * dc[2]));
            const V dchi2 = fma(w[0], dc[0], fma(w[1], dc[1], w[2] * dc[2]));
            // R_ij += (dd_ij + gt_ij tr dd) / (2 chi) - (d_i chi d_j chi + 3 gt_ij |d chi|^2) / (4 chi^2)
            const V tr = hi2 * fma((-3.f * hi2), dchi2, trace(gi, dd));
            const V ca = hi2 * fma(w[0], dal[0], fma(w[1], dal[1], w[2] * dal[2]));
            V n[6];   // -D_i D_j alpha
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const V np = -1.f * p[i];
#pragma unroll
                for (int j = i; j < 3; j++) {
                    const int c = si(i, j);
                    Rc[c] = fma(np, p[j], fma(g[c], tr, fma(hi2, dd[c], Rc[c])));
                    const V s = fma(cu[0][c], dal[0], fma(cu[1][c], dal[1], cu[2][c] * dal[2])) - back(P_T + 14 + c);
                    n[c] = fma(g[c], ca, s - fma(p[i], dal[j], p[j] * dal[i]));
                }
            }
            nlap = chi * trace(gi, n);
#pragma unroll
            for (int c = 0; c < 6; c++) Rc[c] = fma(alpha, Rc[c], n[c]);   // alpha R_ij - D_i D_j alpha so far
        }
        // ---- the connection functions (R_ij += gt_k(i d_j) Gt^k) and K
#pragma unroll 1
        for (int l = 0; l < 4; l++) {
            visit();
            Der<V> d;
            derive<T, PP, false>(tile(v), b, ko, d);
            release();
            keep(l < 3 ? F_GAMX + l : F_K, d.extra);
            keep(l < 3 ? P_GAM + l : P_T + 12, d.q);
#pragma unroll
            for (int j = 0; j < 3; j++) keep(P_T + 3 * l + j, i12h * d.D[j]);
        }
        const V K = back(P_T + 12);
        {
            const V s = (-4.f / 3.f) * alpha, k0 = back(P_T + 9), k1 = back(P_T + 10), k2 = back(P_T + 11);
            const V ha = .5f * alpha;
            V t[6];   // summed by themselves and unscaled: one rounding at the size of the whole
#pragma unroll
            for (int l = 0; l < 3; l++) {
                V e[3];
#pragma unroll
                for (int j = 0; j < 3; j++) e[j] = back(P_T + 3 * l + j);
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = i; j < 3; j++) {
                        const V w = g[si(l, j)] * e[i];
                        t[si(i, j)] = fma(g[si(l, i)], e[j], l == 0 ? w : fma(g[si(l, j)], e[i], t[si(i, j)]));
                    }
            }
#pragma unroll
            for (int c = 0; c < 6; c++) Rc[c] = fma(ha, t[c], Rc[c]);
#pragma unroll
            for (int c = 0; c < 6; c++) keep(P_X + c, Rc[c]);
#pragma unroll
            for (int i = 0; i < 3; i++)   // the connection functions' right-hand side
                keep(P_GC + i, s * fma(gi[si(i, 0)], k0, fma(gi[si(i, 1)], k1, gi[si(i, 2)] * k2)));
        }
        // ---- the trace-free extrinsic curvature (and the shift's driver)
#pragma unroll 1
        for (int l = 0; l < (shift_on ? 9 : 6); l++) {
            visit();
            Der<V> d;
            derive<T, PP, false>(tile(v), b, ko, d);
            release();
            keep(l < 6 ? F_AXX + l : F_BX + (l - 6), d.extra);
            keep(l < 6 ? P_T + l : P_B + (l - 6), d.q);
        }
        V A[6], rA[6], rK;
        {
            V ud[3][3], uu[6], X[6];
#pragma unroll
            for (int c = 0; c < 6; c++) A[c] = back(P_T + c);
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++)
                    ud[i][j] = fma(gi[si(i, 0)], A[si(0, j)], fma(gi[si(i, 1)], A[si(1, j)], gi[si(i, 2)] * A[si(2, j)]));
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = i; j < 3; j++)
                    uu[si(i, j)] = fma(ud[i][0], gi[si(0, j)], fma(ud[i][1], gi[si(1, j)], ud[i][2] * gi[si(2, j)]));
            rK = fma(alpha, fma((1.f / 3.f) * K, K, trace(A, uu)), nlap);
            // gc^i += 2 alpha Gt^i_jk At^jk - At^ij (2 d_j alpha + 3 alpha d_j chi / chi)
            const V a2 = 2.f * alpha, a6 = -6.f * alpha;
            V yv[3];
#pragma unroll
            for (int j = 0; j < 3; j++) yv[j] = fma(a6, p[j], -2.f * dal[j]);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                const V s = fma(a2, trace(uu, cu[i]), back(P_GC + i));
                keep(P_GC + i, fma(uu[si(i, 0)], yv[0], fma(uu[si(i, 1)], yv[1], fma(uu[si(i, 2)], yv[2], s))));
            }
#pragma unroll
            for (int c = 0; c < 6; c++) X[c] = back(P_X + c);
            const V tr = (-1.f / 3.f) * trace(gi, X), aK = alpha * K, na2 = -2.f * alpha;
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = i; j < 3; j++) {
                    const int c = si(i, j);
                    const V s = fma(A[si(i, 0)], ud[0][j], fma(A[si(i, 1)], ud[1][j], A[si(i, 2)] * ud[2][j]));
                    rA[c] = fma(na2, s, fma(aK, A[c], chi * fma(g[c], tr, X[c])));
                }
        }
        // ---- the shift: 12 h d_j beta^l, gt^jk d_j d_k beta^l and d_j d_l beta^l
#pragma unroll 1
        for (int l = 0; l < 3; l++) {
            visit();
            Der<V> d;
            derive<T, PP, true>(tile(v), b, ko, d);
            release();
            keep(F_BETAX + l, shift_on ? d.extra : sp(0.f));
#pragma unroll
            for (int j = 0; j < 3; j++) keep(P_T + 7 * l + j, i12h * d.D[j]);
            keep(P_T + 7 * l + 3, lap(d));
            const V s = -i12h2 * (l == 0 ? d.S[0] : l == 1 ? d.S[1] : d.S[2]);
            const V m0 = i144h2 * (l == 2 ? d.M[1] : d.M[0]), m1 = i144h2 * (l == 0 ? d.M[1] : d.M[2]);
            keep(P_T + 7 * l + 4, l == 0 ? s : m0);
            keep(P_T + 7 * l + 5, l == 1 ? s : (l == 0 ? m0 : m1));
            keep(P_T + 7 * l + 6, l == 2 ? s : m1);
        }
        if (!ok) {   // a wait gave up: report it; the tile's results are dropped
            s_abort = 1;
            atomicExch(a.err, 1);
        }
        if (__any_sync(0xffffffffu, s_abort)) break;
        // ---- the cells of neighbours' ghost layers that hold this cell's values (~0: none)
        uint32_t gx = ~0u, gy = ~0u, gz = ~0u, gxy = ~0u, gxz = ~0u, gyz = ~0u, gxyz = ~0u;
        {
            // from cell `at` of domain `in` to its image in domain `to`, the next along the axis
            auto image = [&](uint32_t at, int32_t in, int axis, int s, int32_t to) -> uint32_t {
                const uint32_t n = axis == 0 ? N : (axis == 1 ? N * T : N * T * T);
                return to < 0 ? ~0u : at + (uint32_t)(to - in) * (T * T * T) + (s == 0 ? n : 0u - n);
            };
            if constexpr (FEED > 0) gx = image(pi, (int32_t)slot, 0, sx, dx);
            if constexpr (FEED > 1) {
                gy = image(pi, (int32_t)slot, 1, sy, dy);
                gxy = image(gx, dx, 1, sy, dxy);
            }
            if constexpr (FEED > 2) {
                gz = image(pi, (int32_t)slot, 2, sz, dz);
                gxz = image(gx, dx, 2, sz, dxz);
                gyz = image(gy, dy, 2, sz, dyz);
                gxyz = image(gxy, dxy, 2, sz, dxyz);
            }
        }
        // tests per field are time where a warp has its scheduler alone (the small tiles): one for most warps
        const bool feeds = (gx & gy & gz & gxy & gxz & gyz & gxyz) != ~0u;
        // ---- right-hand sides, in the fields' order from P_T on
        {
            V rg[6], gc[3], ddb[3], Gam[3];
            const V na2 = -2.f * alpha;
#pragma unroll
            for (int c = 0; c < 6; c++) rg[c] = na2 * A[c];
#pragma unroll
            for (int i = 0; i < 3; i++) {
                Gam[i] = back(P_GAM + i);
                gc[i] = back(P_GC + i) + back(P_T + 7 * i + 3);
                ddb[i] = (1.f / 3.f) * (back(P_T + 4 + i) + back(P_T + 11 + i) + back(P_T + 18 + i));
            }
            V div = sp(0.f);
#pragma unroll
            for (int l = 0; l < 3; l++) {
                V e[3];
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    e[j] = back(P_T + 7 * l + j);
                    gc[l] = gc[l] - Gam[j] * e[j];
                }
                div = div + e[l];
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = i; j < 3; j++) {
                        rg[si(i, j)] = fma(g[si(i, l)], e[j], fma(g[si(j, l)], e[i], rg[si(i, j)]));
                        rA[si(i, j)] = fma(A[si(i, l)], e[j], fma(A[si(j, l)], e[i], rA[si(i, j)]));
                    }
            }
            const V t3 = (-2.f / 3.f) * div, aK = alpha * K;
            keep(P_T + F_CHI, chi * fma(2.f / 3.f, aK, t3));
            keep(P_T + F_K, rK);
            keep(P_T + F_ALPHA, a.prm.slicing == AMR_SLICING_HARMONIC ? (-1.f * alpha) * aK : -2.f * aK);
#pragma unroll
            for (int c = 0; c < 6; c++) {
                keep(P_T + F_GXX + c, fma(g[c], t3, rg[c]));
                keep(P_T + F_AXX + c, fma(A[c], t3, rA[c]));
            }
#pragma unroll
            for (int i = 0; i < 3; i++) {
                gc[i] = gc[i] - Gam[i] * t3;
                gc[i] = fma(gi[si(i, 0)], ddb[0], fma(gi[si(i, 1)], ddb[1], fma(gi[si(i, 2)], ddb[2], gc[i])));
                keep(P_T + F_GAMX + i, gc[i]);
                if (shift_on) {
                    const V B = back(P_B + i);
                    keep(P_T + F_BETAX + i, .75f * B);
                    keep(P_T + F_BX + i, fma(-a.prm.eta, B, gc[i]));
                } else {   // frozen: no right-hand side, no extra term
                    keep(P_T + F_BETAX + i, sp(0.f));
                    keep(P_T + F_BX + i, sp(0.f));
                    keep(F_BX + i, sp(0.f));
                }
            }
        }
        // ---- RK4 stage update.  Stage 1: acc = old + dt/6 k1, out = old + dt/2 k1; 2: acc += dt/3 k2,
        // out = old + dt/2 k2; 3: acc += dt/3 k3, out = old + dt k3; 4: out = acc + dt/6 k4.
        const float dt = a.dt0 / (float)(1u << depth);
        const float c_acc = a.stage == 1 ? dt * (1.f / 6.f) : dt * (1.f / 3.f);
        const float c_out = a.stage == 3 ? dt : (a.stage == 4 ? dt * (1.f / 6.f) : dt * .5f);
        load_own(t + gridDim.x < tiles ? t + gridDim.x : t);   // past the last tile: this one again, unused
        const uint32_t o_old = zl * S::OLD_PLANE + (y + 1) * T + x + 3, o_acc = S::OLD_F + (zl * TY + y) * N + x;
#pragma unroll 1
        for (int u = 0; u < S::UPDATES; u++) {
            visit();
            const float* sl = ring + (size_t)(v % R) * S::SLOT;
            V uo[S::F], ac[S::F];
#pragma unroll
            for (int j = 0; j < S::F; j++) {
                const float* q = sl + j * (S::OLD_F + S::ACC_F);
                uo[j] = V::ld(q + o_old, S::OLD_PLANE);
                ac[j] = V::ld(q + o_acc, TY * N);
            }
            release();
            if (!ok) continue;   // what the slot holds is not this tile's
#pragma unroll
            for (int j = 0; j < S::F; j++) {
                const int f = u * S::F + j;
                const V r = back(P_T + f) + back(f);
                V o;
                if (a.stage == 4) {
                    o = fma(c_out, r, ac[j]);
                } else {
                    const V n = fma(c_acc, r, a.stage == 1 ? uo[j] : ac[j]);
                    n.st(a.acc[f] + ii, N * N);
                    o = fma(c_out, r, uo[j]);
                }
                if (f == F_CHI) o = at_least(o, a.prm.chi_floor - 1.f);   // chi (stored less 1) keeps its floor; a NaN stays
                o.st(a.out[f] + pi, T * T);
                if (FEED > 0 && (L == 2 || feeds)) {
                    float* const to = a.out[f];
                    if (gx != ~0u) o.st(to + gx, T * T);
                    if (FEED > 1 && gy != ~0u) o.st(to + gy, T * T);
                    if (FEED > 1 && gxy != ~0u) o.st(to + gxy, T * T);
                    if (FEED > 2 && zmask) {
                        if (gz != ~0u) o.st(to + gz, T * T, zmask);
                        if (gxz != ~0u) o.st(to + gxz, T * T, zmask);
                        if (gyz != ~0u) o.st(to + gyz, T * T, zmask);
                        if (gxyz != ~0u) o.st(to + gxyz, T * T, zmask);
                    }
                }
            }
        }
        if (!ok) {   // a wait of the update gave up
            s_abort = 1;
            atomicExch(a.err, 1);
        }
        if (__any_sync(0xffffffffu, s_abort)) break;
    }
    // the CTA's shared memory must outlive every copy issued into it: in a normal run all were
    // consumed, after an abort some may be in flight (bounded waits)
    __syncthreads();
    if (tid == 0 && s_abort)
        for (uint32_t n = s_asked, q = n > (uint32_t)R ? n - R : 0u; q < n; q++)
            mbar_wait(&full[q % R], (q / R) & 1u, q + 1u == a.withhold ? spins : kMaxSpins);
}

template <int N, int TY, int TZ, int R_, class V, int MINB, int FEED>
cudaError_t limit_t() {
    static std::atomic<uint64_t> configured{0};
    return ensure_smem_limit(k_evo_stage_bssn<N, TY, TZ, R_, V, MINB, FEED>, StageShape<N, TY, TZ, R_, V::L>::SMEM, configured);
}
template <int N, int TY, int TZ, int R_, class V, int MINB, int FEED>
cudaError_t stage_t(const EvoArgs& a, int sms, cudaStream_t st) {
    using S = StageShape<N, TY, TZ, R_, V::L>;
    const cudaError_t e = limit_t<N, TY, TZ, R_, V, MINB, FEED>();
    if (e != cudaSuccess) return e;
    const uint32_t tiles = a.n_items * (uint32_t)S::TILES, room = (uint32_t)(sms * MINB);
    k_evo_stage_bssn<N, TY, TZ, R_, V, MINB, FEED><<<tiles < room ? tiles : room, S::CT, S::SMEM, st>>>(a);
    return cudaGetLastError();
}

// a substep whose domains are too few to give every SM a large tile (launch_evo_stage_bssn)
bool evo_stage_small(uint32_t n, uint32_t n_batch, int sms) {
    return n == 8u ? n_batch <= (uint32_t)sms : n == 16u && n_batch * 8u <= (uint32_t)sms;
}

}  // namespace

// Axes whose ghost layers a stage writes, for a substep of n_batch domains.  All three where launches count (the
// small tiles, and at 32^3 up to as many domains as at 16^3); along x and y elsewhere, where the z layers'
// stores, N^2 a plane and field all at once, cost more than the fill's pass.  A root step (GB300, cold caches,
// periodic, so that every face is fed) with 0, 1, 2 and 3 axes: 9 domains of 8^3 188, 165, 152, 142 us, 73 492,
// 422, 384, 363, 585 5.14, 4.61, 4.56, 5.49 ms; 9 of 16^3 244, 199, 173, 150 us, 73 1.75, 1.58, 1.53, 1.59 ms,
// 585 24.8, 21.4, 20.7, 22.8; 9 of 32^3 930, 771, 681, 646 us, 73 10.56, 8.99, 8.73, 8.99 ms, 585 164, 137, 134, 140.
int evo_stage_feeds(uint32_t n, uint32_t n_batch) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return evo_stage_small(n == 32u ? 16u : n, n_batch, sms) ? 3 : 2;
}
cudaError_t launch_evo_stage_bssn(const EvoArgs& a, cudaStream_t st) {
    if (a.n_items == 0u) return cudaSuccess;
    if (a.stage < 1 || a.stage > 4) return cudaErrorInvalidValue;
    // The tile: 512 cells of whole planes at 16^3 and 8^3 (one copy a field; 8 rows of two planes at 32^3,
    // where whole planes would be 1024 threads), except where the domains are too few to give every SM
    // such a tile.  Then smaller tiles of one cell a thread, with more CTAs.  A root step (periodic, cold caches, the
    // better number of fed axes on either side), large and small tiles: at 8^3, 9 domains 204 and 142 us,
    // 73 domains 445 and 363, 585 domains 4.57 and 4.75 ms; at 16^3, 9 domains 200 and 150 us, 73 domains
    // 1.53 and 1.85 ms.  A domain of 32^3 has 64 tiles.  The rule reads the substep's domains, not this
    // launch's, so that a domain launched alone rounds as in a batch.
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    switch (a.n) {
        case 8:
            if (evo_stage_small(8, a.n_batch, sms))
                return a.feed ? stage_t<8, 8, 2, 6, V1, 3, 3>(a, sms, st) : stage_t<8, 8, 2, 6, V1, 3, 0>(a, sms, st);
            return stage_t<8, 8, 8, 6, V2, 1, 2>(a, sms, st);
        case 16:
            if (evo_stage_small(16, a.n_batch, sms))
                return a.feed ? stage_t<16, 16, 1, 5, V1, 1, 3>(a, sms, st) : stage_t<16, 16, 1, 5, V1, 1, 0>(a, sms, st);
            return stage_t<16, 16, 2, 6, V2, 1, 2>(a, sms, st);
        case 32: return a.feed_axes == 3 ? stage_t<32, 8, 2, 6, V2, 1, 3>(a, sms, st) : stage_t<32, 8, 2, 6, V2, 1, 2>(a, sms, st);
        default: return cudaErrorInvalidValue;
    }
}
cudaError_t prepare_evo_stage_bssn(uint32_t n) {
    cudaError_t e = cudaErrorInvalidValue;
    switch (n) {
        case 8:
            e = limit_t<8, 8, 2, 6, V1, 3, 3>();
            if (e == cudaSuccess) e = limit_t<8, 8, 2, 6, V1, 3, 0>();
            return e == cudaSuccess ? limit_t<8, 8, 8, 6, V2, 1, 2>() : e;
        case 16:
            e = limit_t<16, 16, 1, 5, V1, 1, 3>();
            if (e == cudaSuccess) e = limit_t<16, 16, 1, 5, V1, 1, 0>();
            return e == cudaSuccess ? limit_t<16, 16, 2, 6, V2, 1, 2>() : e;
        case 32:
            e = limit_t<32, 8, 2, 6, V2, 1, 3>();
            return e == cudaSuccess ? limit_t<32, 8, 2, 6, V2, 1, 2>() : e;
        default: return e;
    }
}

}  // namespace amr
