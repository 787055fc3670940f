// Fused MR-LBM time step: stream + moment evaluation + collision in one pass over HBM (one moment
// read, one moment write per node).
//
// Replaces the reference's two full-grid kernels and their population halo
// (paths inside sakthi-lbm/MRLBM_3D_CUDA):
//   streaming_and_evaluate_Mom  MRLBM_3D/src/solver/mlbm.cu:83-164
//   collision_halo_update       MRLBM_3D/src/solver/mlbm.cu:186-242
//   pop_load_from_halo / pop_save_to_halo / save_pop / streaming
//                               MRLBM_3D/src/core/D3Q27/halo_interface.cuh:5-201, core/streaming.cuh:6-35
// The reference streams populations rebuilt from the stored (post-collision) moments,
// f_q(x) = R(M(x - c_q))_q on a grid that wraps in every axis, then evaluates moments, then
// collides.  Here a node's 27 pulled populations never leave registers: a lane owns two nodes
// x, x + 1 of a row (every operation in packed FP32, sm_100's .f32x2), and its warp
//   y: reads the stored moments of the rows y + 1, y, y - 1 of a plane from shared memory and rebuilds
//      the nine populations of each that enter row y (c_y = -1, 0, +1);
//   x: takes the neighbours' across lanes by shuffles;
//   z: sums each c_z class of the plane (row and column sums) and marches along z with the classes
//      of two planes in registers.
// A row is rebuilt three times (139 packed operations a lane instead of 80), but no population crosses
// shared memory and no warp waits for another: only the copies of the rows' moments are shared.
// Bound by issue and FP32 throughput with 16-bit storage (600 warp instructions per 64 nodes, 65% of the
// issue slots), by issue and HBM with FP32 storage (54%, 5.8 TB/s).  256^3 on GB300, before (populations exchanged
// through shared-memory rings between CTA barriers) and now: FP32 335 -> 231 us a step, FP16 283 -> 206,
// hybrid 298 -> 216, BF16 283 -> 213.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <string>

#include "mrlbm_internal.h"
#include "packed.cuh"
#include "storage.cuh"

namespace mrlbm {
namespace {

// A CTA owns a column of TILE_X x TY nodes and marches along z.  (TY = 32, for grids of at most 32 nodes along x: a
// tile is 32 rows of one x-block, an owner warp holds two rows, 16 lanes each, and a row wraps within
// itself, so there are no side columns and no halo values.  In 64-node tiles half the lanes or more are idle there:
// 32 x 512 x 512 194 us a step in FP32 and 212 in FP16, in such tiles 108 and 107; 8 x 1024 x 1024 709 -> 336.)
//   owner warps (one per row): lane l owns the nodes x0 + 2 l and x0 + 2 l + 1;
//   halo warps (every NH-th plane each): issue the bulk copies of a plane's rows (own columns, rows
//     y0 - 1 .. y0 + TY) into a ring of D plane stages, and evaluate the x-pass values that enter the
//     tile from the columns x0 - 1 and x0 + TILE_X (one lane per row and side), up to D planes
//     ahead of the owners.
// A stage is full when its copies have landed and its halo values are written (mbarrier full[s]: the
// copies' bytes and one arrival) and free again when every owner warp has read it (empty[s], one
// arrival per owner warp); owners drift apart freely within the ring.  The sequence of stages runs on
// from one work item to the next, so there is no drain between items.
template <typename S, int TY, bool SPECIAL>
struct Geo {
    static constexpr bool NARROW = TY == 32;
    static constexpr int RPW = NARROW ? 2 : 1;               // rows of one owner warp
    static constexpr int OW = TY / RPW;                      // owner warps
    static constexpr int XW = TILE_X / RPW;                  // nodes of one row
    static constexpr int WPN = StorageLayout<S>::words;      // 32-bit words of one node
    static constexpr int ROWW = XW * WPN;                    // words of one row (one or two x-blocks)
    static constexpr int SIDEC = NARROW ? 0 : 2 * (TY + 2);  // columns beside the tile, corners included
    static constexpr int MARKW = SPECIAL ? TY * XW / 4 : 0;  // node marks of the plane, a byte each
    static constexpr int STAGEW = (TY + 2) * ROWW + SIDEC * WPN + MARKW;  // words of one plane stage
    // Stages, and class sums parked in shared memory between planes (all nine class sums and the c_z = +1
    // class do not fit the owners' 104 registers).  Shared memory and L1 share 256 KB, and the owners'
    // remaining spills need L1: FP32 256^3 takes 240 us with 3 stages and 3 parked sums (164 KB, 92 KB of L1),
    // 254 us with 6 parked, 285 us with 4 stages (28 KB of L1: 336 us); all with stores through L1, 232 us now.
    // (FP32 tiles of 8 rows, two CTAs an SM: 410 us with 4 stages each, 327 with 3.)
    static constexpr int D = OW == 16 ? (WPN == 10 ? 3 : (WPN == 7 ? 4 : 5)) : (WPN == 10 ? (TY == 8 ? 3 : 4) : (WPN == 7 ? 5 : 6));
    static constexpr int PARK = OW != 16 ? 0 : (WPN == 10 ? 3 : 6);
    static constexpr int HALO = NARROW ? 0 : 9;              // floats per row and side: c_y x c_z
    static constexpr int NH = OW / 4;                        // halo warps
    static constexpr int NTH = 32 * (OW + NH);
    // 20 warps share 16,384 registers per scheduler: 96 each at launch (640 x 96 = 61,440), then 104 for the
    // four warpgroups of owners and 64 for the halo warps (512 x 104 + 128 x 64 = 61,440)
    static constexpr bool SPLIT = OW == 16;
    static constexpr int MINB = TY == 4 ? 3 : (TY == 8 ? 2 : 1);  // resident CTAs per SM targeted
    static constexpr int SMEM = D * (STAGEW * 4 + 2 * TY * HALO * 4 + 3 * 8 + 16) + PARK * 32 * OW * 8;
    static_assert(NARROW || 2 * TY <= 32, "one halo lane per row and side");
    static_assert(STAGEW % 4 == 0 && ROWW % 4 == 0 && (SIDEC * WPN) % 4 == 0 && (2 * TY * HALO) % 4 == 0 && MARKW % 4 == 0,
                  "bulk copies and 16-byte accesses on 16-byte boundaries");
};

// Constants of the rebuild for stored u s_u, m s_m, (rho - rho0) s_r.
struct RebuildK {
    float rho0, ir;             // 1 / s_r
    float h3, h15, h45, h9;     // Hermite factors 3 / s_u, 1.5 / s_m, 4.5 / s_m, 9 / s_m
};
template <typename S>
__device__ __forceinline__ RebuildK rebuild_k(float rho0, const StorageScale &sc) {
    if constexpr (std::is_same<S, float>::value) return {rho0, 1.0f, 3.0f, 1.5f, 4.5f, 9.0f};
    else
        return {rho0, sc.is[0], __fmul_rn(3.0f, sc.is[1]), __fmul_rn(1.5f, sc.is[2]), __fmul_rn(4.5f, sc.is[2]),
                __fmul_rn(9.0f, sc.is[2])};
}

// Ten stored values of one node (float) or of the two nodes of a lane (V2).
template <typename T>
struct Stored {
    T r, ux, uy, uz, mxx, myy, mzz, mxy, mxz, myz;
};

__host__ __device__ constexpr int direction(int cx, int cy, int cz) {
    for (int q = 0; q < 27; ++q)
        if (cxq(q) == cx && cyq(q) == cy && czq(q) == cz) return q;
    return -1;
}

// The sign bits of both lanes.
__device__ __forceinline__ float negated(float a) { return -a; }
__device__ __forceinline__ V2 negated(V2 a) { return V2{a.v ^ 0x8000000080000000ull}; }

// Populations of one node (float) or of a lane's two (V2) from the stored moments: reconstruct_h of
// lbm_device.cuh, operation by operation, in units of their weight class.  The weights are 16, 4, 1 and
// 1/4 times w = 1/54 (as floats too), and a power of two commutes with every rounding, so
//   f[0] / 16, f[1..6] / 4, f[7..18], 4 f[19..26]
// all come from r = w rho; the sums below put the factors back.  The caller's unused populations fold
// away.
static_assert(kW0 == 16.0f * kW2 && kW1 == 4.0f * kW2 && 4.0f * kW3 == kW2, "weights are powers of two apart");
template <typename S, typename T>
__device__ __forceinline__ void rebuild_scaled(const Stored<T> &m, const RebuildK &k, T f[27]) {
    const T rho = kScaled<S> ? fma(m.r, bc<T>(k.ir), bc<T>(k.rho0)) : add(bc<T>(k.rho0), m.r);
    const T t = add(add(m.mxx, m.myy), m.mzz);
    const T h45 = bc<T>(k.h45);
    const T p0 = fma(bc<T>(-k.h15), t, bc<T>(1.0f));
    const T ax = fma(h45, m.mxx, p0), ay = fma(h45, m.myy, p0);
    const T r = mul(rho, bc<T>(kW2)), q = mul(bc<T>(k.h3), r), n = mul(bc<T>(k.h9), r);
    const T nq = negated(q), nn = negated(n);
    f[0] = mul(r, p0);
    {
        const T ex = mul(r, ax), ey = mul(r, ay), ez = mul(r, fma(h45, m.mzz, p0));
        f[1] = fma(q, m.ux, ex);
        f[2] = fma(nq, m.ux, ex);
        f[3] = fma(q, m.uy, ey);
        f[4] = fma(nq, m.uy, ey);
        f[5] = fma(q, m.uz, ez);
        f[6] = fma(nq, m.uz, ez);
    }
    const T upp = add(m.ux, m.uy), upm = sub(m.ux, m.uy);
    {
        const T b = mul(r, fma(h45, m.myy, ax));
        const T cp = fma(n, m.mxy, b), cm = fma(nn, m.mxy, b);
        f[7] = fma(q, upp, cp);
        f[8] = fma(nq, upp, cp);
        f[13] = fma(q, upm, cm);
        f[14] = fma(nq, upm, cm);
    }
    {
        const T b = mul(r, fma(h45, m.mzz, ax));
        const T cp = fma(n, m.mxz, b), cm = fma(nn, m.mxz, b);
        const T sp = add(m.ux, m.uz), sm = sub(m.ux, m.uz);
        f[9] = fma(q, sp, cp);
        f[10] = fma(nq, sp, cp);
        f[15] = fma(q, sm, cm);
        f[16] = fma(nq, sm, cm);
    }
    {
        const T b = mul(r, fma(h45, m.mzz, ay));
        const T cp = fma(n, m.myz, b), cm = fma(nn, m.myz, b);
        const T sp = add(m.uy, m.uz), sm = sub(m.uy, m.uz);
        f[11] = fma(q, sp, cp);
        f[12] = fma(nq, sp, cp);
        f[17] = fma(q, sm, cm);
        f[18] = fma(nq, sm, cm);
    }
    {
        const T c0 = mul(r, fma(h45, t, p0));
        const T a = add(m.mxy, m.mxz), b = sub(m.mxy, m.mxz);
        const T e1 = fma(n, add(a, m.myz), c0), e2 = fma(n, sub(b, m.myz), c0);
        const T e3 = fma(nn, add(b, m.myz), c0), e4 = fma(nn, sub(a, m.myz), c0);
        const T u1 = add(upp, m.uz), u2 = sub(upp, m.uz), u3 = add(upm, m.uz), u4 = sub(upm, m.uz);
        f[19] = fma(q, u1, e1);
        f[20] = fma(nq, u1, e1);
        f[21] = fma(q, u2, e2);
        f[22] = fma(nq, u2, e2);
        f[23] = fma(q, u3, e3);
        f[24] = fma(nq, u3, e3);
        f[26] = fma(q, u4, e4);
        f[25] = fma(nq, u4, e4);
    }
}

// Stored values of the lane's two nodes from a row in shared memory (`p`: the lane's first word).
template <typename S>
__device__ __forceinline__ Stored<V2> load_pair(const uint32_t *p) {
    Stored<V2> m;
    if constexpr (std::is_same<S, float>::value) {
        V2 w[10];
#pragma unroll
        for (int f = 0; f < 10; ++f) w[f].v = *reinterpret_cast<const unsigned long long *>(p + f * kXBlock);
        m = {w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], w[8], w[9]};
    } else if constexpr (kHybrid<S>) {
        V2 u[3];
#pragma unroll
        for (int f = 0; f < 3; ++f) u[f].v = *reinterpret_cast<const unsigned long long *>(p + f * kXBlock);
        float2 a[4], b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint2 w = *reinterpret_cast<const uint2 *>(p + (3 + j) * kXBlock);
            a[j] = pair_to_f<__half>(w.x);
            b[j] = pair_to_f<__half>(w.y);
        }
        m = {v2(a[0].x, b[0].x), u[0], u[1], u[2], v2(a[0].y, b[0].y), v2(a[1].x, b[1].x), v2(a[1].y, b[1].y),
             v2(a[2].x, b[2].x), v2(a[2].y, b[2].y), v2(a[3].x, b[3].x)};
    } else {
        float2 a[5], b[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            const uint2 w = *reinterpret_cast<const uint2 *>(p + j * kXBlock);
            a[j] = pair_to_f<S>(w.x);
            b[j] = pair_to_f<S>(w.y);
        }
        m = {v2(a[0].x, b[0].x), v2(a[0].y, b[0].y), v2(a[1].x, b[1].x), v2(a[1].y, b[1].y), v2(a[2].x, b[2].x),
             v2(a[2].y, b[2].y), v2(a[3].x, b[3].x), v2(a[3].y, b[3].y), v2(a[4].x, b[4].x), v2(a[4].y, b[4].y)};
    }
    return m;
}

// Stored values of one side column (words SIDEC apart).
template <typename S, int SIDEC>
__device__ __forceinline__ Stored<float> side_values(const uint32_t *p) {
    Raw<S> raw;
    load_raw_words<S, SIDEC>(p, raw);
    float v[10];
    raw_values<S>(raw, v);
    return {v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9]};
}

// Sums of one c_z class over (c_x, c_y): orders 1, c_x, c_y, c_x^2, c_y^2, c_x c_y (the classes c_z = +-1
// times 4: their populations are in units of a quarter).
struct ClassSums {
    V2 s0, sx, sy, sxx, syy, sxy;
};

// Post-stream moments of a lane's two nodes: rho - rho0, and u, m with their storage scales.
struct Pair {
    V2 r, ux, uy, uz, mxx, myy, mzz, mxy, mxz, myz;
};

struct Node {
    float r, ux, uy, uz, mxx, myy, mzz, mxy, mxz, myz;
};
__device__ __forceinline__ Node node_of(const Pair &p, int c) {
    return c == 0 ? Node{lo(p.r), lo(p.ux), lo(p.uy), lo(p.uz), lo(p.mxx), lo(p.myy), lo(p.mzz), lo(p.mxy), lo(p.mxz), lo(p.myz)}
                  : Node{hi(p.r), hi(p.ux), hi(p.uy), hi(p.uz), hi(p.mxx), hi(p.myy), hi(p.mzz), hi(p.mxy), hi(p.mxz), hi(p.myz)};
}

// m_ab <- (1 - omega) m_ab + omega u_a u_b on scaled moments (collide_h on two nodes).
__device__ __forceinline__ void collide_pair(Pair &m, float omega, float omega_u) {
    const V2 om1 = bc<V2>(1.0f - omega), ou = bc<V2>(omega_u);
    const V2 wx = mul(ou, m.ux), wy = mul(ou, m.uy), wz = mul(ou, m.uz);
    m.mxx = fma(wx, m.ux, mul(om1, m.mxx));
    m.myy = fma(wy, m.uy, mul(om1, m.myy));
    m.mzz = fma(wz, m.uz, mul(om1, m.mzz));
    m.mxy = fma(wx, m.uy, mul(om1, m.mxy));
    m.mxz = fma(wx, m.uz, mul(om1, m.mxz));
    m.myz = fma(wy, m.uz, mul(om1, m.myz));
}

// The stored words of one node (r: rho - rho0, u and m already scaled); key: random bits of a
// stochastically rounded store.
template <typename S, bool SR>
__device__ __forceinline__ void node_words(const Node &m, float sr, uint32_t key, uint32_t w[]) {
    if constexpr (std::is_same<S, float>::value) {
        const float v[10] = {m.r, m.ux, m.uy, m.uz, m.mxx, m.myy, m.mzz, m.mxy, m.mxz, m.myz};
#pragma unroll
        for (int f = 0; f < 10; ++f) w[f] = __float_as_uint(v[f]);
    } else {
        const float r = m.r * sr;
        if constexpr (kHybrid<S>) {
            w[0] = __float_as_uint(m.ux);
            w[1] = __float_as_uint(m.uy);
            w[2] = __float_as_uint(m.uz);
            w[3] = round_pair<__half, SR>(r, m.mxx, key, 0);
            w[4] = round_pair<__half, SR>(m.myy, m.mzz, key, 1);
            w[5] = round_pair<__half, SR>(m.mxy, m.mxz, key, 2);
            w[6] = round_pair<__half, SR>(m.myz, 0.0f, key, 3);
        } else {
            w[0] = round_pair<S, SR>(r, m.ux, key, 0);
            w[1] = round_pair<S, SR>(m.uy, m.uz, key, 1);
            w[2] = round_pair<S, SR>(m.mxx, m.myy, key, 2);
            w[3] = round_pair<S, SR>(m.mzz, m.mxy, key, 3);
            w[4] = round_pair<S, SR>(m.mxz, m.myz, key, 4);
        }
    }
}

// The collided moments leave past L1 (UNCACHED), which is then left to what the owners spill: FP32 at 256^3
// 240.6 -> 232.5 us a step, an FP32 annulus 250 -> 240, a cylinder wake in hybrid storage 363 -> 349.  Plain
// hybrid tiles spill nothing that comes back and are 1 % slower so (218 -> 221): they store as usual.
template <typename S, bool SR, bool UNCACHED>
__device__ __forceinline__ void store_pair(uint32_t *p, const Pair &m, float sr, uint32_t key0, uint32_t key1) {
    constexpr int WPN = StorageLayout<S>::words;
    uint32_t a[WPN], b[WPN];
    node_words<S, SR>(node_of(m, 0), sr, key0, a);
    node_words<S, SR>(node_of(m, 1), sr, key1, b);
#pragma unroll
    for (int f = 0; f < WPN; ++f) {
        if constexpr (UNCACHED) store_uncached(p + f * kXBlock, a[f], b[f]);
        else *reinterpret_cast<uint2 *>(p + f * kXBlock) = make_uint2(a[f], b[f]);
    }
}
template <typename S, bool SR>
__device__ __forceinline__ void store_node(uint32_t *p, const Node &m, float sr, uint32_t key) {
    constexpr int WPN = StorageLayout<S>::words;
    uint32_t a[WPN];
    node_words<S, SR>(m, sr, key, a);
#pragma unroll
    for (int f = 0; f < WPN; ++f) store_uncached(p + f * kXBlock, a[f]);
}

// Post-stream (pre-collision) moments of a wall-stencil node into its side-buffer entry, the
// snapshot the wall kernel interpolates from (the node-list kernel writes the same for the
// marked nodes it handles); iu / im undo the storage scales.
__device__ __forceinline__ void snapshot(float *e, const Node &m, float iu, float im) {
    store_side(e, m.r, m.ux * iu, m.uy * iu, m.uz * iu, m.mxx * im, m.myy * im, m.mzz * im, m.mxy * im, m.mxz * im,
               m.myz * im);
}

// Storage word of node x = 32 xb (a block's first node) of row y, plane z.
template <typename S>
__device__ __forceinline__ int64_t row_word(int xb, int y, int z, int nxb, int ny) {
    return ((((int64_t)z * ny + y) * nxb + xb) * StorageLayout<S>::words) * kXBlock;
}

// SPECIAL = false: every node of every item is a plain bulk node (no node marks are read).  Four 128^3 boxes in a
// batch, with and without SPECIAL: FP32 178 and 155 us a step, FP16 167 and 142.
template <typename S, int TY, bool SPECIAL, bool BATCH>
__global__ void __launch_bounds__(Geo<S, TY, SPECIAL>::NTH, Geo<S, TY, SPECIAL>::MINB)
    step_kernel(const __grid_constant__ StepArgs single, const BatchArgs *__restrict__ ba, const int parity,
                double *__restrict__ diag_part) {
    using G = Geo<S, TY, SPECIAL>;
    constexpr bool TAKEOVER = SPECIAL || BATCH;
    extern __shared__ __align__(128) unsigned char smem[];
    uint32_t *const stages = reinterpret_cast<uint32_t *>(smem);
    float *const halos = reinterpret_cast<float *>(smem + G::D * G::STAGEW * 4);
    // {case, work item, its number} of the item that starts with the stage's plane
    int4 *const heads = reinterpret_cast<int4 *>(smem + G::D * (G::STAGEW * 4 + 2 * TY * G::HALO * 4));
    uint64_t *const full = reinterpret_cast<uint64_t *>(heads + G::D);
    uint64_t *const empty = full + G::D;
    uint64_t *const landed = empty + G::D;
    V2 *const park = reinterpret_cast<V2 *>(landed + G::D) + threadIdx.x;  // owners: the thread's slots, 32 OW apart
    __shared__ __align__(16) uint4 s_slot[2];  // answers to takeover requests, by item parity
    __shared__ uint64_t s_taken;
    __shared__ int s_next[2];
    __shared__ int s_failed;  // 1 + the plane at which a halo warp's wait ran out: none is issued from there on

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < G::D; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, G::OW);
            mbar_init(landed + s, 1);
        }
        mbar_init(&s_taken, 1);
        s_failed = 0;
        mbar_init_fence();
    }
    __syncthreads();
    int stage = 0;
    uint32_t phase = 0;
    auto next_stage = [&]() {
        if (++stage == G::D) {
            stage = 0;
            phase ^= 1u;
        }
    };
    const int n_items = BATCH ? ba->n_items : single.n_items;
    const int limit = BATCH ? ba->cases[0]->wait_limit : single.wait_limit;
    // a wait ran out: which items are left undone is not known, so every case of a batch has it
    auto report = [&]() {
        if constexpr (BATCH)
            for (int c = 0; c < ba->n_cases; ++c) atomicOr_system(ba->cases[c]->error, kErrorWait);
        else
            atomicOr_system(single.error, kErrorWait);
    };

    if (warp >= G::OW) {
        if constexpr (G::SPLIT) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        // ---- halo warps ------------------------------------------------------------------------
        bool ok = true;
        const int hw = warp - G::OW;
        int q = 0;        // planes so far, over all items: plane q is halo warp q % NH's
        int n = 0;        // items so far
        auto take_turn = [&]() {
            if (G::NH > 1 && q > 0) token_wait(3 + hw);
            if (!ok) return;
            volatile int *const failed = &s_failed;
            ok = (G::NH == 1 || *failed == 0) && mbar_wait(empty + stage, phase ^ 1u, limit);
            if (!ok && lane == 0 && *failed == 0) *failed = q + 1;
        };
        // Work items.  TAKEOVER: one CTA per item is launched, and a CTA that finishes its item takes over
        // one that has not started (tiles with boundary nodes and the cases of a batch cost unevenly).
        // Otherwise the CTAs stride through the items.
        const bool leader = threadIdx.x == 32 * G::OW;
        for (int it = blockIdx.x; it >= 0 && it < n_items;) {
            int2 head;
            if constexpr (BATCH) head = ba->items[it];
            else head = make_int2(0, single.items ? single.items[it] : (it % (single.tiles_x * single.tiles_y)) |
                                                                       ((it / (single.tiles_x * single.tiles_y)) << 20));
            const StepArgs &a = BATCH ? *ba->cases[head.x] : single;
            const int nx = a.nx, ny = a.ny, nz = a.nz, nxb = a.nxb;
            const uint32_t *__restrict__ src = reinterpret_cast<const uint32_t *>(a.m[parity]);
            const RebuildK K = rebuild_k<S>(a.rho0, a.sc);
            const int tile = head.y & 0xFFFFF, seg = head.y >> 20;
            const int tix = tile % a.tiles_x, tiy = tile / a.tiles_x;
            const int x0 = tix * G::XW, y0 = tiy * TY;
            const int w = min(G::XW, nx - x0), h = min(TY, ny - y0);
            const int zs = seg * a.lz, ze = min(zs + a.lz, nz), last = ze - zs + 1;
            const int64_t zst = (int64_t)ny * nxb * G::WPN * kXBlock;
            auto wrap = [](int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); };
            // rows of the bulk copies: lane r copies row y0 - 1 + r (and row y0 + 31 + r)
            const uint32_t row_bytes = (uint32_t)min(2, nxb - 2 * tix) * G::WPN * kXBlock * 4;
            auto copies = [&](int r) { return r < h + 2; };
            auto row_off = [&](int r) { return copies(r) ? row_word<S>(2 * tix, wrap(y0 - 1 + r, ny), 0, nxb, ny) : (int64_t)0; };
            const int64_t copy_off = row_off(lane), copy_off2 = G::NARROW ? row_off(lane + 32) : 0;
            // node marks of the planes that this segment updates (row by row)
            const uint32_t mark_pitch = (uint32_t)a.tiles_x * TILE_X;
            const uint8_t *marks = SPECIAL && lane < h && a.tile_slot && a.tile_slot[tile] >= 0
                                       ? a.mark + ((int64_t)zs * ny + y0 + lane) * mark_pitch + x0
                                       : nullptr;
            const bool tile_marked = SPECIAL && __shfl_sync(0xffffffffu, marks != nullptr, 0);
            auto marked = [&](int k) { return tile_marked && k >= 1 && k < last; };
            // columns beside the tile: column c = side * (TY + 2) + row + 1 is
            // x0 - 1 (side 0, entering with c_x = +1) or x0 + w (side 1), rows -1 .. h; lane c fetches
            // column c, and the columns past the 32nd are spread over the lanes
            auto side_column = [&](int c) {
                if (G::NARROW) return (int64_t)-1;
                const int sd = c / (TY + 2), r = c - sd * (TY + 2) - 1;
                if (sd > 1 || r > h) return (int64_t)-1;
                const int gx = wrap(sd ? x0 + w : x0 - 1, nx);
                return row_word<S>(gx >> 5, wrap(y0 + r, ny), 0, nxb, ny) + (gx & 31);
            };
            const int64_t col_off = side_column(lane);
            constexpr int EXTRA = G::SIDEC > 32 ? G::SIDEC - 32 : 0;  // 4 for 16 rows
            constexpr int NE = EXTRA ? EXTRA : 1, PER = 32 / NE;  // words of such a column fetched per round
            const int64_t ext_off = EXTRA ? side_column(32 + lane % NE) : -1;
            const int side = lane / TY, row = lane - side * TY;  // the column this lane evaluates
            const bool active = !G::NARROW && side < 2 && row < h;
            const int mine = (hw + G::NH - q % G::NH) % G::NH;  // this warp's first plane of the item
            int zk = (zs == 0 ? nz - 1 : zs - 1) + mine;
            if (zk >= nz) zk -= nz;
            // The next item is asked for as the last planes of this one are issued: the answer is there before
            // their stages are free, and an item whose CTA is only late (the node-list kernel's blocks are in
            // its place) is not put behind this one's whole length (an annulus of 132 items: 321 -> 265 us a step).
            if (TAKEOVER && leader && mine > last) takeover_request(s_slot + (n & 1), &s_taken);
            for (int k = 0; k <= last; ++k, ++q, next_stage()) {
                if ((k - mine) % G::NH != 0) continue;
                if (TAKEOVER && leader && k + G::NH > last) takeover_request(s_slot + (n & 1), &s_taken);
                // The halo warps wait for a free stage in turn, each asleep at a hardware barrier until the one
                // before it has passed (polling costs issue slots).  Plane q waits for the release of plane
                // q - D; the turn before has seen that of q - 1 - D, so the release two uses back on the stage
                // is past, which the one parity bit of the wait could not tell from the last one.  For that, no
                // turn succeeds after one that failed.
                take_turn();
                if (G::NH > 1) token_pass(3 + (hw + 1) % G::NH);
                if (!ok) continue;
                uint32_t *const sp = stages + stage * G::STAGEW;
                uint32_t *const cp = sp + (TY + 2) * G::ROWW;  // [word][column]
                if (lane == 0) {
                    if (k == 0) heads[stage] = make_int4(head.x, head.y, it, 0);
                    mbar_expect_tx(landed + stage, row_bytes * (h + 2) + (marked(k) ? G::XW * (uint32_t)h : 0u));
                    mbar_arrive(landed + stage);
                }
                __syncwarp();
                const uint32_t *const zsrc = src + zk * zst;
                if (copies(lane)) bulk_load(sp + lane * G::ROWW, zsrc + copy_off, row_bytes, landed + stage);
                if (G::NARROW && copies(lane + 32))
                    bulk_load(sp + (lane + 32) * G::ROWW, zsrc + copy_off2, row_bytes, landed + stage);
                if (marked(k) && lane < h)
                    bulk_load(cp + G::SIDEC * G::WPN + lane * (G::XW / 4), marks + (int64_t)(k - 1) * ny * mark_pitch, G::XW,
                              landed + stage);
                if constexpr (!G::NARROW) {
                    // (not through L1: a line per word would push out what the owners spill)
                    uint32_t w0[G::WPN], w1[(G::WPN + PER - 1) / PER];
                    if (col_off >= 0) {
#pragma unroll
                        for (int f = 0; f < G::WPN; ++f) w0[f] = load_uncached(zsrc + col_off + f * kXBlock);
                    }
                    if (EXTRA && ext_off >= 0) {
#pragma unroll
                        for (int i = 0; i < (G::WPN + PER - 1) / PER; ++i) {
                            const int f = i * PER + lane / NE;
                            if (f < G::WPN) w1[i] = load_uncached(zsrc + ext_off + f * kXBlock);
                        }
                    }
                    if (col_off >= 0) {
#pragma unroll
                        for (int f = 0; f < G::WPN; ++f) cp[f * G::SIDEC + lane] = w0[f];
                    }
                    if (EXTRA && ext_off >= 0) {
#pragma unroll
                        for (int i = 0; i < (G::WPN + PER - 1) / PER; ++i) {
                            const int f = i * PER + lane / NE;
                            if (f < G::WPN) cp[f * G::SIDEC + 32 + lane % NE] = w1[i];
                        }
                    }
                }
                __syncwarp();
                zk += G::NH;
                while (zk >= nz) zk -= nz;
                if constexpr (!G::NARROW) {
                    if (active) {
                        float *e = halos + ((stage * 2 + side) * TY + row) * G::HALO;
#pragma unroll
                        for (int cy = -1; cy <= 1; ++cy) {
                            float f[27];
                            rebuild_scaled<S>(side_values<S, G::SIDEC>(cp + side * (TY + 2) + row + 1 - cy), K, f);
#pragma unroll
                            for (int cz = -1; cz <= 1; ++cz)
                                e[3 * (cy + 1) + cz + 1] = side ? f[direction(-1, cy, cz)] : f[direction(1, cy, cz)];
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full + stage);
                }
            }
            if constexpr (TAKEOVER) {
                // one answer for all halo warps (two slots: the next one is written a barrier after the
                // last read of this one)
                if (leader) {
                    const bool answered = mbar_wait_lane(&s_taken, n & 1);
                    s_next[n & 1] = answered ? takeover_result(s_slot + (n & 1)) : -1;
                    if (!answered && s_failed == 0) *(volatile int *)&s_failed = q + 1;
                }
                asm volatile("bar.sync 2, %0;" ::"r"(32 * G::NH) : "memory");
                it = s_next[n & 1];
                if (*(const volatile int *)&s_failed) ok = false;
                ++n;
            } else {
                it += (int)gridDim.x;
            }
        }
        if (q % G::NH == hw) {
            take_turn();
            if (ok && lane == 0) {
                heads[stage] = make_int4(0, -1, 0, 0);  // end mark: plane q
                mbar_arrive(landed + stage);
                if (!G::NARROW) mbar_arrive(full + stage);
            }
        }
        if (!ok && lane == 0) report();
        // The CTA stays until its copies have landed, also when a wait ran out and its owners are gone: the
        // shared memory that they fill would be the next CTA's.  No halo warp issues another one past the
        // barrier; all planes before the failed one were issued (or all, and the end mark), and the last D
        // are the stages' last uses, under way or the last that ended, so their parities tell.
        asm volatile("bar.sync 2, %0;" ::"r"(32 * G::NH) : "memory");
        if (threadIdx.x == 32 * G::OW) {
            const int issued = s_failed ? s_failed - 1 : q + 1;
            for (int p = max(0, issued - G::D); p < issued; ++p) mbar_wait_lane(landed + p % G::D, (uint32_t)(p / G::D) & 1u);
        }
    } else {
        if constexpr (G::SPLIT) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        // ---- owner warps -----------------------------------------------------------------------
        bool ok = limit > 0;  // 0: the first wait has run out
        int items = 0;
        while (ok) {
            // landed before full, here and in every plane: rows past the tile's last one skip the waits on
            // full, and only the landing of a stage (its refill follows the release of its last use) makes
            // the one parity bit of that wait unambiguous
            ok = mbar_wait(landed + stage, phase, limit) && (G::NARROW || mbar_wait(full + stage, phase, limit));
            if (!ok) break;
            const int4 head = heads[stage];
            if (head.y < 0) break;
            const StepArgs &a = BATCH ? *ba->cases[head.x] : single;
            const int nx = a.nx, ny = a.ny, nxb = a.nxb;
            const RebuildK K = rebuild_k<S>(a.rho0, a.sc);
            const int tile = head.y & 0xFFFFF, seg = head.y >> 20;
            const int tix = tile % a.tiles_x, tiy = tile / a.tiles_x;
            const int x0 = tix * G::XW, y0 = tiy * TY;
            const int w = min(G::XW, nx - x0), h = min(TY, ny - y0);
            const int zs = seg * a.lz, ze = min(zs + a.lz, a.nz), last = ze - zs + 1;
            // the lane's row of the tile, and its place in the row
            const int row = G::NARROW ? 2 * warp + (lane >> 4) : warp, at = G::NARROW ? lane & 15 : lane;
            const int y = y0 + row, x = x0 + 2 * at;
            const bool own = row < h && 2 * at < w;
            const int last_lane = (w >> 1) - 1;
            // (two rows a warp) the lanes of the x-neighbours in a row that wraps
            const int west = at == 0 ? lane + last_lane : lane - 1, east = at == last_lane ? lane - at : lane + 1;
            const int64_t zst = (int64_t)ny * nxb * G::WPN * kXBlock;
            const int in_row = (G::NARROW ? 0 : (lane >> 4) * (G::WPN * kXBlock)) + 2 * (lane & 15);  // the lane's word in a row
            uint32_t *dst = reinterpret_cast<uint32_t *>(a.m[parity ^ 1]) + row_word<S>(2 * tix, y, zs, nxb, ny) + in_row;
            const float su = kScaled<S> ? a.sc.s[1] : 1.0f, sm = kScaled<S> ? a.sc.s[2] : 1.0f;
            const float iu = kScaled<S> ? a.sc.is[1] : 1.0f, im = kScaled<S> ? a.sc.is[2] : 1.0f;
            const float omega = a.omega, omega_u = kScaled<S> ? a.omega * (sm * (iu * iu)) : a.omega;
            const float cs = kScaled<S> ? __fmul_rn(-kCs2, sm) : -kCs2;
            const bool sr_on = kScaled<S> && a.sr_step != nullptr;
            const uint32_t sr_seed = sr_on ? sr_step_seed(*a.sr_step) : 0u;
            const int slot = SPECIAL && a.tile_slot ? a.tile_slot[tile] : -1;  // -1: no boundary nodes
            float *side = SPECIAL ? a.side + side_index(slot, x, y, zs, x0, y0, a.nz, TILE_X, TY) * 16 : nullptr;
            uint32_t marks = 0u;  // of the lane's nodes in plane k - 1, a byte each
            float dm = 0.f, de = 0.f;
            volatile float totals[2];  // of sampled steps: kept on the stack, not in registers

            // times 4, of the plane emitted next: sums of its c_z = +1 and 0 classes (c_z = +1 from the plane
            // below), and of its c_z = +1 class alone; c_z = +1 class of the plane read last
            V2 pr, px, py, pxx, pyy, pxy, u0s, uxs, uys;
            ClassSums up;
            pr.v = px.v = py.v = pxx.v = pyy.v = pxy.v = u0s.v = uxs.v = uys.v = 0ull;
            up = {pr, pr, pr, pr, pr, pr};

            // store the collided moments of the lane's nodes (u0, u1: which of them) in plane z
            constexpr bool UNCACHED = SPECIAL || !kHybrid<S>;
            auto put = [&](uint32_t *p, const Pair &o, bool u0, bool u1, int z) {
                const float sr = a.sc.s[0];
                if (sr_on) {
                    const uint32_t k0 = sr_key(sr_seed, x, y, z, nx, ny), k1 = sr_key(sr_seed, x + 1, y, z, nx, ny);
                    if (u0 && u1) store_pair<S, true, UNCACHED>(p, o, sr, k0, k1);
                    else if (u0 || u1) store_node<S, true>(p + !u0, node_of(o, u0 ? 0 : 1), sr, u0 ? k0 : k1);
                } else {
                    if (u0 && u1) store_pair<S, false, UNCACHED>(p, o, sr, 0u, 0u);
                    else if (u0 || u1) store_node<S, false>(p + !u0, node_of(o, u0 ? 0 : 1), sr, 0u);
                }
            };
            auto plane = [&](const int k) {
                if (k > 0 && ok) ok = mbar_wait(landed + stage, phase, limit);
                if (!ok) return;
                Pair o;
                V2 rho4;  // 4 rho, as the sums in `o`
                uint32_t marks_in = 0u;
                if (G::RPW * warp < h) {  // (a tile has whole pairs of rows: ny is a multiple of 8)
                    const uint32_t *sp = stages + stage * G::STAGEW + row * G::ROWW + in_row;
                    const float *hv = halos + ((stage * 2 + (lane >= 16 || lane == last_lane)) * TY + warp) * G::HALO;
                    // the nine populations of the row y - cy that enter this row, shifted along x;
                    // g[cx + 1][cz + 1]
                    auto pulled = [&](auto cyc, V2 (&g)[3][3]) {
                        constexpr int cy = decltype(cyc)::value;
                        V2 f[27];
                        rebuild_scaled<S>(load_pair<S>(sp + (1 - cy) * G::ROWW), K, f);
                        if constexpr (G::NARROW) {
#pragma unroll
                            for (int c = 0; c < 3; ++c) {
                                const V2 fp = f[direction(1, cy, c - 1)], fm = f[direction(-1, cy, c - 1)];
                                g[2][c] = v2(__shfl_sync(0xffffffffu, hi(fp), west), lo(fp));
                                g[1][c] = f[direction(0, cy, c - 1)];
                                g[0][c] = v2(hi(fm), __shfl_sync(0xffffffffu, lo(fm), east));
                            }
                            return;
                        }
                        // the side columns' populations are evaluated meanwhile
                        if (cy == -1 && k > 0) ok = mbar_wait(full + stage, phase, limit);
                        const float e[3] = {hv[3 * (cy + 1)], hv[3 * (cy + 1) + 1], hv[3 * (cy + 1) + 2]};
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const V2 fp = f[direction(1, cy, c - 1)], fm = f[direction(-1, cy, c - 1)];
                            const float left = __shfl_up_sync(0xffffffffu, hi(fp), 1);
                            const float right = __shfl_down_sync(0xffffffffu, lo(fm), 1);
                            g[2][c] = v2(lane == 0 ? e[c] : left, lo(fp));
                            g[1][c] = f[direction(0, cy, c - 1)];
                            g[0][c] = v2(hi(fm), lane == last_lane ? e[c] : right);
                        }
                    };
                    // row by row into each class's row and column sums (c_y = -1, 0, +1), where a population
                    // with one zero less among (c_x, c_y) weighs 4 times as much
                    const V2 four = bc<V2>(4.0f);
                    V2 mm[3], pm[3], rm[3], cm[3], cp[3], r0[3], g[3][3];
                    pulled(std::integral_constant<int, -1>{}, g);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        mm[c] = g[0][c];
                        pm[c] = g[2][c];
                        rm[c] = add(fma(g[1][c], four, g[0][c]), g[2][c]);
                    }
                    pulled(std::integral_constant<int, 0>{}, g);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        r0[c] = add(fma(g[1][c], four, g[0][c]), g[2][c]);  // a quarter of it
                        cp[c] = fma(g[2][c], four, pm[c]);
                        cm[c] = fma(g[0][c], four, mm[c]);
                    }
                    if constexpr (SPECIAL) {
                        // a solid node of an updated block keeps its stored moments, collided (the reference
                        // collides every node of an active block); a plain fluid node whose only mark is the
                        // wall-stencil bit is updated like any bulk node, plus its snapshot; every other
                        // marked node is the node-list kernel's, or frozen
                        if (slot >= 0 && own && k >= 1 && k < last)
                            marks_in = *reinterpret_cast<const uint16_t *>(
                                reinterpret_cast<const uint8_t *>(stages + stage * G::STAGEW + (TY + 2) * G::ROWW + G::SIDEC * G::WPN) +
                                row * G::XW + 2 * at);
                        const bool q0 = marks_in & MARK_SOLID, q1 = marks_in & (MARK_SOLID << 8);
                        if (q0 || q1) {
                            const Stored<V2> q = load_pair<S>(sp + G::ROWW);
                            // unscaled, collided and scaled again, as the reference order rounds it
                            Pair so{q.r, q.ux, q.uy, q.uz, q.mxx, q.myy, q.mzz, q.mxy, q.mxz, q.myz};
                            auto rescale = [&](V2 u, V2 v) {
                                for (V2 *p : {&so.ux, &so.uy, &so.uz}) *p = mul(*p, u);
                                for (V2 *p : {&so.mxx, &so.myy, &so.mzz, &so.mxy, &so.mxz, &so.myz}) *p = mul(*p, v);
                            };
                            if constexpr (kScaled<S>) {
                                so.r = sub(fma(q.r, bc<V2>(K.ir), bc<V2>(K.rho0)), bc<V2>(K.rho0));
                                rescale(bc<V2>(iu), bc<V2>(im));
                            }
                            float *const e = side + (int64_t)(k - 1) * (TILE_X * TY * 16);
                            if (q0 && (marks_in & MARK_SNAPSHOT)) snapshot(e, node_of(so, 0), 1.0f, 1.0f);
                            if (q1 && (marks_in & (MARK_SNAPSHOT << 8))) snapshot(e + 16, node_of(so, 1), 1.0f, 1.0f);
                            collide_pair(so, omega, omega);
                            if constexpr (kScaled<S>) rescale(bc<V2>(su), bc<V2>(sm));
                            put(dst + (k >= 2 ? zst : 0), so, q0, q1, zs + k - 1);
                        }
                    }
                    pulled(std::integral_constant<int, 1>{}, g);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty + stage);
                    auto finish = [&](int c) {
                        const V2 rp = add(fma(g[1][c], four, g[0][c]), g[2][c]);
                        const V2 cpc = add(cp[c], g[2][c]), cmc = add(cm[c], g[0][c]);
                        return ClassSums{add(fma(r0[c], four, rp), rm[c]), sub(cpc, cmc), sub(rp, rm[c]), add(cpc, cmc), add(rp, rm[c]),
                                         sub(add(g[2][c], mm[c]), add(pm[c], g[0][c]))};
                    };
                    const ClassSums dn = finish(0);
                    {
                        V2 *const v[] = {&uys, &uxs, &pxy, &pyy, &pxx, &u0s, &py, &px, &pr};
#pragma unroll
                        for (int i = 0; i < G::PARK; ++i) *v[i] = park[i * 32 * G::OW];
                    }
                    rho4 = add(pr, dn.s0);
                    o.ux = add(px, dn.sx);
                    o.uy = add(py, dn.sy);
                    o.uz = sub(u0s, dn.s0);
                    o.mxx = add(pxx, dn.sxx);
                    o.myy = add(pyy, dn.syy);
                    o.mzz = add(u0s, dn.s0);
                    o.mxy = add(pxy, dn.sxy);
                    o.mxz = sub(uxs, dn.sx);
                    o.myz = sub(uys, dn.sy);
                    const ClassSums flat = finish(1);
                    pr = fma(flat.s0, four, up.s0);
                    px = fma(flat.sx, four, up.sx);
                    py = fma(flat.sy, four, up.sy);
                    pxx = fma(flat.sxx, four, up.sxx);
                    pyy = fma(flat.syy, four, up.syy);
                    pxy = fma(flat.sxy, four, up.sxy);
                    u0s = up.s0;
                    uxs = up.sx;
                    uys = up.sy;
                    {
                        V2 *const v[] = {&uys, &uxs, &pxy, &pyy, &pxx, &u0s, &py, &px, &pr};
#pragma unroll
                        for (int i = 0; i < G::PARK; ++i) park[i * 32 * G::OW] = *v[i];
                    }
                    up = finish(2);
                } else {
                    // rows past the tile's last one read nothing but the stage's head, all lanes before the release
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty + stage);
                }
                next_stage();
                if (k >= 2) {
                    if (own) {
                        const V2 rho = mul(rho4, bc<V2>(0.25f));
                        const V2 inv = v2(__frcp_rn(lo(rho)), __frcp_rn(hi(rho)));  // correctly rounded
                        const V2 vu = mul(inv, bc<V2>(0.25f * su)), vm = kScaled<S> ? mul(inv, bc<V2>(0.25f * sm)) : vu;
                        o.r = sub(rho, bc<V2>(a.rho0));
                        o.ux = mul(o.ux, vu);
                        o.uy = mul(o.uy, vu);
                        o.uz = mul(o.uz, vu);
                        o.mxx = fma(o.mxx, vm, bc<V2>(cs));
                        o.myy = fma(o.myy, vm, bc<V2>(cs));
                        o.mzz = fma(o.mzz, vm, bc<V2>(cs));
                        o.mxy = mul(o.mxy, vm);
                        o.mxz = mul(o.mxz, vm);
                        o.myz = mul(o.myz, vm);
                        bool u0 = true, u1 = true;  // nodes updated here
                        if constexpr (SPECIAL) {
                            u0 = !(marks & MARK_OTHER);
                            u1 = !(marks & (MARK_OTHER << 8));
                            float *const e = side + (int64_t)(k - 2) * (TILE_X * TY * 16);
                            if (u0 && (marks & MARK_SNAPSHOT)) snapshot(e, node_of(o, 0), iu, im);
                            if (u1 && (marks & (MARK_SNAPSHOT << 8))) snapshot(e + 16, node_of(o, 1), iu, im);
                        }
                        if (!BATCH && diag_part) {
                            const float ke = 0.5f * (iu * iu);
                            const V2 e2 = fma(o.ux, o.ux, fma(o.uy, o.uy, mul(o.uz, o.uz)));
                            dm += (u0 ? lo(o.r) : 0.f) + (u1 ? hi(o.r) : 0.f);
                            de += ke * ((u0 ? lo(e2) : 0.f) + (u1 ? hi(e2) : 0.f));
                        }
                        collide_pair(o, omega, omega_u);
                        put(dst, o, u0, u1, zs + k - 2);
                    }
                    dst += zst;
                }
                marks = marks_in;
            };
            // every 16 planes of a sampled step the lane's sums go to its running totals: no FP32 sum runs over a long
            // segment (over 2 x 256 equal terms, added node by node, it drifted by up to 94 x 2^-24)
            const bool sampled = !BATCH && diag_part != nullptr;
            auto to_totals = [&](bool first) {
                totals[0] = first ? dm : totals[0] + dm;
                totals[1] = first ? de : totals[1] + de;
                dm = de = 0.f;
            };
            // The loop in two shapes, each where it is the faster one: 256^3, plane by plane FP32 230 us a step (a
            // sampled one 246), FP16 215 (228); by runs of planes FP32 233 (256), FP16 207 (219).
            if constexpr (G::WPN == 10) {
#pragma unroll 1
                for (int k = 0; k <= last && ok; ++k) {
                    plane(k);
                    if (sampled && k > 1 && (k == last || (k & 15) == 1)) to_totals(k <= 17);  // plane k - 2 was emitted
                }
            } else {
#pragma unroll 1
                for (int k = 0; k <= last && ok;) {
                    const bool first = k == 0;
                    const int stop = sampled ? min(last + 1, first ? 18 : k + 16) : last + 1;
#pragma unroll 1
                    for (; k < stop && ok; ++k) plane(k);
                    if (sampled) to_totals(first);
                }
            }
            if (sampled) {
                // the warp's sums over the item -> their slot of diag_part (items of a strided launch that
                // share a CTA share its slots, in order): the same sums whichever CTA takes the item
                double dmD = (double)totals[0], deD = (double)totals[1];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    dmD += __shfl_down_sync(0xffffffffu, dmD, o);
                    deD += __shfl_down_sync(0xffffffffu, deD, o);
                }
                if (lane == 0) {
                    const int at = (SPECIAL ? head.z : (int)blockIdx.x) * G::OW + warp;
                    if (!SPECIAL && items > 0) {
                        dmD += diag_part[2 * at + 0];
                        deD += diag_part[2 * at + 1];
                    }
                    diag_part[2 * at + 0] = dmD;
                    diag_part[2 * at + 1] = deD;
                }
                ++items;
            }
        }
        if (!ok && lane == 0) report();
    }
}

__global__ void diag_finalize_kernel(const double *__restrict__ part, int n, double *__restrict__ out,
                                     int *__restrict__ error) {
    __shared__ double s[2][256];
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        a += part[2 * i];
        b += part[2 * i + 1];
    }
    s[0][threadIdx.x] = a;
    s[1][threadIdx.x] = b;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            s[0][threadIdx.x] += s[0][threadIdx.x + o];
            s[1][threadIdx.x] += s[1][threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = s[0][0];
        out[1] = s[1][0];
        if (error && !(isfinite(s[0][0]) && isfinite(s[1][0]))) atomicOr(error, kErrorDiverged);
    }
}

// Opt the kernel into its dynamic shared memory once per device (the attribute belongs to the
// current device's context; never set inside a stream capture: batched launches are prepared
// before their graphs are captured).  Devices past the 64th are configured on every launch.
template <typename S, int TY, bool SP, bool BATCH>
cudaError_t configure_t() {
    static std::atomic<unsigned long long> configured{0ull};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (bit && (configured.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    if constexpr (Geo<S, TY, SP>::SPLIT) {
        // the register split hands out exactly what the launch allocates: refuse a build whose launch
        // allocates less (the owners would wait for registers that never come)
        cudaFuncAttributes at;
        if ((e = cudaFuncGetAttributes(&at, step_kernel<S, TY, SP, BATCH>)) != cudaSuccess) return e;
        if ((at.numRegs + 7) / 8 * 8 * Geo<S, TY, SP>::NTH <
            32 * (Geo<S, TY, SP>::OW * 104 + Geo<S, TY, SP>::NH * 64))
            return cudaErrorLaunchOutOfResources;
    }
    e = cudaFuncSetAttribute(step_kernel<S, TY, SP, BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             Geo<S, TY, SP>::SMEM);
    if (e != cudaSuccess) return e;
    configured.fetch_or(bit, std::memory_order_acq_rel);
    return cudaSuccess;
}

template <typename S, int TY, bool SP, bool BATCH>
cudaError_t launch_t(const StepArgs &a, const BatchArgs *ba, int parity, double *diag_part, int n_ctas, cudaStream_t s,
                     cudaEvent_t placed = nullptr) {
    const cudaError_t e = configure_t<S, TY, SP, BATCH>();
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeLaunchCompletionEvent;
    at[0].val.launchCompletionEvent.event = placed;
    at[0].val.launchCompletionEvent.flags = 0;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(n_ctas);
    c.blockDim = dim3(Geo<S, TY, SP>::NTH);
    c.dynamicSmemBytes = Geo<S, TY, SP>::SMEM;
    c.stream = s;
    c.attrs = at;
    c.numAttrs = placed ? 1 : 0;
    return cudaLaunchKernelEx(&c, step_kernel<S, TY, SP, BATCH>, a, ba, parity, diag_part);
}

// Run f(storage type tag, tile-height tag) for the storage mode and tile height.
template <typename T>
struct Tag {
    using type = T;
};
template <typename F>
auto dispatch(int storage, int tile_y, F f) -> decltype(f(Tag<float>{}, std::integral_constant<int, 4>{})) {
    auto height = [&](auto tag) {
        switch (tile_y) {
            case 4: return f(tag, std::integral_constant<int, 4>{});
            case 8: return f(tag, std::integral_constant<int, 8>{});
            case 32: return f(tag, std::integral_constant<int, 32>{});
            default: return f(tag, std::integral_constant<int, 16>{});
        }
    };
    switch (storage) {
        case MRLBM_STORAGE_F16: return height(Tag<__half>{});
        case MRLBM_STORAGE_BF16: return height(Tag<__nv_bfloat16>{});
        case MRLBM_STORAGE_F16_U32: return height(Tag<HybridWord>{});
        default: return height(Tag<float>{});
    }
}
bool known(int storage, int tile_y) {
    return storage >= MRLBM_STORAGE_F32 && storage <= MRLBM_STORAGE_F16_U32 && (tile_y == 4 || tile_y == 8 || tile_y == 16 || tile_y == 32);
}

}  // namespace

cudaError_t launch_step(const StepLaunch &l, int storage, int tile_y, bool special, cudaStream_t s) {
    if (!known(storage, tile_y)) return cudaErrorInvalidValue;
    return dispatch(storage, tile_y, [&](auto t, auto ty) {
        using S = typename decltype(t)::type;
        return special ? launch_t<S, ty(), true, false>(*l.args, nullptr, l.parity, l.diag_part, l.n_ctas, s, l.placed)
                       : launch_t<S, ty(), false, false>(*l.args, nullptr, l.parity, l.diag_part, l.n_ctas, s, l.placed);
    });
}

// (batches of plain cases have a kernel of their own for the default tiles only)
cudaError_t prepare_step_batch(int storage, int tile_y, bool special) {
    if (!known(storage, tile_y)) return cudaErrorInvalidValue;
    return dispatch(storage, tile_y, [&](auto t, auto ty) {
        using S = typename decltype(t)::type;
        if constexpr (ty() >= 16)
            if (!special) return configure_t<S, ty(), false, true>();
        return configure_t<S, ty(), true, true>();
    });
}

cudaError_t launch_step_batch(const BatchArgs *ba, int parity, int storage, int tile_y, bool special, int n_items,
                              cudaStream_t s) {
    if (!known(storage, tile_y)) return cudaErrorInvalidValue;
    return dispatch(storage, tile_y, [&](auto t, auto ty) {
        using S = typename decltype(t)::type;
        if constexpr (ty() >= 16)
            if (!special) return launch_t<S, ty(), false, true>(StepArgs(), ba, parity, nullptr, n_items, s);
        return launch_t<S, ty(), true, true>(StepArgs(), ba, parity, nullptr, n_items, s);
    });
}

cudaError_t launch_diag_finalize(const double *part, int n, double *out, int *error, cudaStream_t s) {
    diag_finalize_kernel<<<1, 256, 0, s>>>(part, n, out, error);
    return cudaGetLastError();
}

int step_kernel_max_ctas_per_sm(int storage, int tile_y) {
    if (!known(storage, tile_y)) return 0;
    return dispatch(storage, tile_y, [&](auto t, auto ty) {
        using S = typename decltype(t)::type;
        int n = 0;
        if (configure_t<S, ty(), true, false>() != cudaSuccess) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, step_kernel<S, ty(), true, false>, Geo<S, ty(), true>::NTH,
                                                          Geo<S, ty(), true>::SMEM) != cudaSuccess)
            return 0;
        return n;
    });
}

// A work item of l planes costs about 2 l + 7 units (of half a plane: filling and draining its pipeline is
// the 7).  The node-list kernel runs beside the step kernel on the SMs that have no item, its rest after
// it: 0.03 units of an SM per node in FP32 (annulus: 196 k nodes, 69 us on 152 SMs, a unit 1.56 us),
// less with fewer words a node, and a block's latency of 5 units at least.  With that term a channel of 32
// planes takes l = 3 instead of 2 (9 us of 40 less a step), an annulus of 256 planes 52 (43: 10 us of 247 more, 24: 16,
// 64: 15, 32: 19).
int choose_lz(int nx, int ny, int nz, int storage, int tile_y, int64_t slots, int active, int list_nodes) {
    const int64_t tiles = active > 0 ? active : (int64_t)((nx + TILE_X - 1) / TILE_X) * ((ny + tile_y - 1) / tile_y);
    const double list = (storage == MRLBM_STORAGE_F32 ? 0.03 : (storage == MRLBM_STORAGE_F16_U32 ? 0.024 : 0.02)) * list_nodes;
    double best = 1e300;
    int lz = nz;
    // each segment length once, with the fewest segments that give it
    for (int nseg = 1; nseg <= std::min(nz, kMaxSegments);) {
        const int l = (nz + nseg - 1) / nseg;
        const int64_t items = tiles * ((nz + l - 1) / l), t = (items + slots - 1) / slots * (2 * l + 7);
        const double rest = list - (double)(slots * t - items * (2 * l + 7));
        const double cost = (double)t + (rest > 0.0 ? std::max(rest / (double)slots, 5.0) : 0.0);
        if (cost < best) {
            best = cost;
            lz = l;
        }
        if (l == 1) break;
        nseg = (nz + l - 2) / (l - 1);
    }
    return lz;
}

// A batch has many more items than the SMs hold, and a CTA takes the next one as it finishes: the items'
// total counts (long segments), and half of the longest as the tail.
int choose_batch_lz(const std::vector<int> &tiles, const std::vector<int> &nz, int storage, int n_sm, int ty) {
    const double slots = (double)std::max(1, step_kernel_max_ctas_per_sm(storage, ty)) * n_sm;
    const int top = *std::max_element(nz.begin(), nz.end());
    double best = 1e300;
    int lz = top;
    // (a work item holds 11 bits of segment: no more segments than that for the tallest case)
    for (int l = (top + kMaxSegments - 1) / kMaxSegments; l <= top; ++l) {
        double work = 0.0;
        for (size_t c = 0; c < nz.size(); ++c) {
            const int seg = (nz[c] + l - 1) / l;
            work += (double)tiles[c] * (2.0 * nz[c] + 7.0 * seg);
        }
        const double cost = work / slots + 0.5 * (2.0 * l + 7.0);
        if (cost < best) {
            best = cost;
            lz = l;
        }
    }
    return lz;
}

// ---- allocation-free periodic step --------------------------------------------------------
// For callers that cannot allocate device memory: what a step needs besides the caller's buffers
// (diagnostics partials and sums) lives in this fixed array of the library's device image, laid out
// as in kernels.h; the argument block travels with the launch.  Every call that asks for
// diagnostics shares the array: such calls race on it when they overlap on the GPU (two streams, or
// two host threads).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
// Error word of each device's calls, in managed memory: set by a kernel whose wait ran out, and read by the
// host without a copy or a synchronisation, so that a call without diagnostics (which returns before its
// kernel has run) is reported by the next one.
static __managed__ int g_noalloc_error[kNoAllocMaxDevices];

namespace {

std::mutex g_noalloc_mu;
// per device, set up on its first call: the scratch array's device address, the error word, and how many CTAs of
// the plain FP32 step kernel it holds with tiles of 16 and of 32 rows
struct NoAllocDevice {
    void *scratch = nullptr;
    int *error = nullptr;
    int slots[2] = {0, 0};
};
NoAllocDevice g_noalloc_dev[kNoAllocMaxDevices];

// CTAs of the plain FP32 step kernel that an SM holds (0: a query failed).
template <int TY>
int plain_ctas_per_sm() {
    int n = 0;
    if (configure_t<float, TY, false, false>() != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, step_kernel<float, TY, false, false>, Geo<float, TY, false>::NTH,
                                                      Geo<float, TY, false>::SMEM) != cudaSuccess)
        return 0;
    return n;
}

// Set-up of device `dev` (the current device), once: the arrays' addresses (in host code the scratch
// array's name is only a host-side stand-in) and the CTAs it holds.  Host-side queries only; nothing is
// allocated.
cudaError_t noalloc_device(int dev, NoAllocDevice &out) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    NoAllocDevice &d = g_noalloc_dev[dev];
    if (!d.scratch) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        void *w = nullptr;
        if ((e = cudaGetSymbolAddress(&w, g_noalloc_error)) != cudaSuccess) return e;
        int n_sm = 0;
        if ((e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        for (int k = 0; k < 2; ++k) {
            const int per_sm = k ? plain_ctas_per_sm<32>() : plain_ctas_per_sm<16>();
            if (per_sm <= 0) return cudaErrorLaunchOutOfResources;
            d.slots[k] = per_sm * n_sm;
        }
        d.error = (int *)w + dev;
        d.scratch = p;
    }
    out = d;
    return cudaSuccess;
}

int noalloc_cuda_fail(cudaError_t e, const char *what, std::string &err) {
    err = std::string("mrlbm_step_periodic_noalloc: ") + what + ": " + cudaGetErrorString(e);
    return e == cudaErrorNoKernelImageForDevice ? MRLBM_ERR_UNSUPPORTED : MRLBM_ERR_CUDA;
}

// Whether a kernel has set the error word; clears it.
bool noalloc_take_error(const NoAllocDevice &d) {
    return __atomic_load_n(d.error, __ATOMIC_ACQUIRE) != 0 && __atomic_exchange_n(d.error, 0, __ATOMIC_ACQ_REL) != 0;
}

}  // namespace

int noalloc_periodic_step(const NoAllocStep &p, std::string &err) {
    const char *fn = "mrlbm_step_periodic_noalloc: ";
    // host-side checks first: nothing below runs for a rejected call
    if (!p.m_in || !p.m_out) {
        err = std::string(fn) + "null moment buffer";
        return MRLBM_ERR_INVALID_ARG;
    }
    if (p.nx <= 0 || p.ny <= 0 || p.nz <= 0 || p.nx % 8 || p.ny % 8 || p.nz % 4) {
        err = std::string(fn) + "grid must be positive multiples of 8 x 8 x 4";
        return MRLBM_ERR_INVALID_ARG;
    }
    if ((int64_t)p.nx * p.ny * p.nz >= (1LL << 31) * 8) {
        err = std::string(fn) + "grid too large";
        return MRLBM_ERR_INVALID_ARG;
    }
    if (!(p.omega > 0.f && p.omega < 2.f) || !(p.rho0 > 0.f) || !std::isfinite(p.rho0)) {
        err = std::string(fn) + "need 0 < omega < 2 and rho0 > 0";
        return MRLBM_ERR_INVALID_ARG;
    }
    if ((uintptr_t)p.m_in % 16 || (uintptr_t)p.m_out % 16) {
        err = std::string(fn) + "moment buffers must be 16-byte aligned";
        return MRLBM_ERR_INVALID_ARG;
    }
    const int64_t bytes = aos_elements(p.nx, p.ny, p.nz) * (int64_t)sizeof(float);
    const uintptr_t a = (uintptr_t)p.m_in, b = (uintptr_t)p.m_out;
    if ((a <= b ? b - a : a - b) < (uint64_t)bytes) {
        err = std::string(fn) + "input and output moment buffers overlap";
        return MRLBM_ERR_INVALID_ARG;
    }
    const int64_t patches = (int64_t)((p.nx + 31) / 32) * ((p.ny + 15) / 16);
    if (patches > kNoAllocMaxTiles) {
        err = std::string(fn) + "grid too large for the fixed 64 KiB scratch: " + std::to_string(patches) +
              " xy tiles of 32 x 16 nodes, at most " + std::to_string(kNoAllocMaxTiles);
        return MRLBM_ERR_INVALID_ARG;
    }

    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return noalloc_cuda_fail(e, "cudaGetDevice", err);
    if (dev < 0 || dev >= kNoAllocMaxDevices) {
        err = std::string(fn) + "device ordinal out of range";
        return MRLBM_ERR_UNSUPPORTED;
    }
    NoAllocDevice nd;
    if (!g_noalloc_dev[dev].scratch) {
        int major = 0, minor = 0;
        if ((e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev)) != cudaSuccess)
            return noalloc_cuda_fail(e, "cudaDeviceGetAttribute", err);
        if (!(major == 10 && minor == 3)) {
            err = std::string(fn) + "libmrlbm is built for sm_103a (GB300) only";
            return MRLBM_ERR_UNSUPPORTED;
        }
    }
    if ((e = noalloc_device(dev, nd)) != cudaSuccess) return noalloc_cuda_fail(e, "device set-up", err);
    if (noalloc_take_error(nd)) {
        err = std::string(fn) + "a wait inside the step kernel of an earlier call ran out: that call's output is not complete "
                                "(this call has launched nothing)";
        return MRLBM_ERR_TIMEOUT;
    }
    unsigned char *scratch = (unsigned char *)nd.scratch;

    const int ty = tile_height(p.nx, 0), slots = nd.slots[ty == 32];
    const int lz = choose_lz(p.nx, p.ny, p.nz, MRLBM_STORAGE_F32, ty, slots);
    const int tiles_x = (p.nx + TILE_X - 1) / TILE_X, tiles_y = (p.ny + ty - 1) / ty;
    const int n_items = tiles_x * tiles_y * ((p.nz + lz - 1) / lz);
    const int n_ctas = std::min(std::min(n_items, slots), kNoAllocMaxParts / owner_warps(ty));

    StepArgs sa;
    sa.m[0] = const_cast<float *>(p.m_in);
    sa.m[1] = p.m_out;
    sa.nxb = (p.nx + kXBlock - 1) / kXBlock;
    sa.n_items = n_items;  // no list: item i is tile i % tiles of segment i / tiles
    sa.nx = p.nx;
    sa.ny = p.ny;
    sa.nz = p.nz;
    sa.tiles_x = tiles_x;
    sa.tiles_y = tiles_y;
    sa.tile_y = ty;
    sa.lz = lz;
    sa.omega = p.omega;
    sa.rho0 = p.rho0;
    for (int k = 0; k < 3; ++k) sa.sc.s[k] = sa.sc.is[k] = 1.f;
    sa.error = nd.error;
    sa.wait_limit = p.wait_limit;
    double *part = (double *)(scratch + kNoAllocPartOffset);
    double *sums = (double *)(scratch + kNoAllocDiagOffset);
    StepLaunch L;
    L.args = &sa;
    L.n_ctas = n_ctas;
    L.diag_part = p.diag_host ? part : nullptr;
    if ((e = launch_step(L, MRLBM_STORAGE_F32, ty, false, p.stream)) != cudaSuccess)
        return noalloc_cuda_fail(e, "step launch", err);
    if (p.diag_host) {
        if ((e = launch_diag_finalize(part, n_ctas * owner_warps(ty), sums, nullptr, p.stream)) != cudaSuccess)
            return noalloc_cuda_fail(e, "diagnostics launch", err);
        double v[2];
        if ((e = cudaMemcpyAsync(v, sums, sizeof(v), cudaMemcpyDeviceToHost, p.stream)) != cudaSuccess ||
            (e = cudaStreamSynchronize(p.stream)) != cudaSuccess)
            return noalloc_cuda_fail(e, "diagnostics read-back", err);
        if (noalloc_take_error(nd)) {
            err = std::string(fn) + "a wait inside the step kernel ran out";
            return MRLBM_ERR_TIMEOUT;
        }
        p.diag_host[0] = (double)p.nx * p.ny * p.nz * p.rho0 + v[0];
        p.diag_host[1] = v[1];
        if (!std::isfinite(v[0]) || !std::isfinite(v[1])) {
            err = std::string(fn) + "mass / energy diagnostics are not finite";
            return MRLBM_ERR_DIVERGED;
        }
    }
    return MRLBM_OK;
}

}  // namespace mrlbm
