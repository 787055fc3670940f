// Boundary and other non-bulk nodes, from a list, beside the step kernel: three lanes a node gather its
// populations, then one applies the closure.
//
// The step kernel updates every plain bulk node in its fused pass, including plain fluid nodes
// whose only mark is the wall-stencil bit (it also writes their snapshot), and collides the solid
// nodes of updated blocks in place.  Every other node that carries a node word (domain faces /
// edges / corners, BCFLUID, BCSOLID, curved-wall nodes) is this kernel's: its closure needs single
// populations, rebuilt here from the stored moments of its neighbours; then it snapshots stencil
// nodes for the wall kernel, collides and stores.
// It reads the state before the step only, so it runs beside the step kernel.  Nodes of blocks
// the reference never updates (frozen) are in no list.
// Bound by the latency of scattered loads (197 k nodes of an annulus: 196 MB of HBM traffic in 67 us, 34% of the
// issue slots, 15 warps an SM); all nine rows of a node are loaded at once for that reason.
//
// Reference (paths inside sakthi-lbm/MRLBM_3D_CUDA):
//   evaluate_bounday_moments dispatch   MRLBM_3D/src/solver/mlbm.cu:166-184
//   cylinder_boundary_moments / annulus_boundary_moments
//                                       MRLBM_3D/src/cases/cylinder/cylinder_kernels.cuh:32-65,
//                                       MRLBM_3D/src/cases/annulus/annulus_kernels.cuh:17-58
//   boundary_condition (faces, edges, corners), fluid_boundary_condition (BCFLUID),
//   bcsolid_boundary_condition (BCSOLID, z walls only)
//                                       MRLBM_3D/src/cases/cylinder/boundaries.cuh:8-1214
//   evaluate_incoming_moments_rotated   MRLBM_3D/src/boundary/curvedLBM.cu:5-59
//   moment_collision                    MRLBM_3D/src/solver/mlbm.cu:3-16
//   compute_force_mass_kernel (BCFLUID part)  MRLBM_3D/src/statistics/forces.cu:25-133
#include <type_traits>

#include "mrlbm_internal.h"
#include "storage.cuh"

namespace mrlbm {
namespace {

// Density and velocity from a full set of 27 populations.
__device__ __forceinline__ Mom rho_u_of(const float *f) {
    float r = 0.f, jx = 0.f, jy = 0.f, jz = 0.f;
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        r += f[q];
        jx += f[q] * (float)cxq(q);
        jy += f[q] * (float)cyq(q);
        jz += f[q] * (float)czq(q);
    }
    Mom m;
    const float inv = 1.0f / r;
    m.rho = r;
    m.ux = jx * inv;
    m.uy = jy * inv;
    m.uz = jz * inv;
    m.mxx = m.myy = m.mzz = m.mxy = m.mxz = m.myz = 0.f;
    return m;
}

// Post-stream density and velocity of node (x, y, z): its 27 populations pulled from the
// stored moments of the neighbours, on the grid that wraps in every axis.
template <typename S>
__device__ __noinline__ Mom pulled_rho_u(const StepArgs &a, const S *__restrict__ src, int x, int y, int z) {
    float f[27];
#pragma unroll 1
    for (int q = 0; q < 27; ++q) {
        const int xs = (x - cxq(q) + a.nx) % a.nx, ys = (y - cyq(q) + a.ny) % a.ny, zs = (z - czq(q) + a.nz) % a.nz;
        float raw[10], g[27];
        load_raw<S>(src, aos_at<S>(xs, ys, zs, a.nxb, a.ny), raw);
        rebuild<S>(raw, a.rho0, a.sc, g);
        f[q] = g[q];
    }
    return rho_u_of(f);
}

__host__ __device__ constexpr int direction(int cx, int cy, int cz) {
    for (int q = 0; q < 27; ++q)
        if (cxq(q) == cx && cyq(q) == cy && czq(q) == cz) return q;
    return -1;
}

// One population f_(cx, CY, CZ) from the stored values of its node, cx at run time: reconstruct_h, whose
// populations all have the form W [fma(q, s, fma(n, c, r E))] with s = (cx ux + CY uy) + CZ uz and
// c = (cx CY mxy + cx CZ mxz) + CY CZ myz.  Signs and zeros are exact, and the weights are powers of two
// apart (as floats too), so this rounds as reconstruct_h does in all 27 cases.
static_assert(kW0 == 16.0f * kW2 && kW1 == 4.0f * kW2 && 4.0f * kW3 == kW2, "weights are powers of two apart");
template <typename S, int CY, int CZ>
__device__ __forceinline__ float population(const float v[10], int cx, float rho0, const StorageScale &sc) {
    const bool f32 = std::is_same<S, float>::value;
    const float h3 = f32 ? 3.0f : __fmul_rn(3.0f, sc.is[1]), h15 = f32 ? 1.5f : __fmul_rn(1.5f, sc.is[2]);
    const float h45 = f32 ? 4.5f : __fmul_rn(4.5f, sc.is[2]), h9 = f32 ? 9.0f : __fmul_rn(9.0f, sc.is[2]);
    const float rho = f32 ? __fadd_rn(rho0, v[0]) : __fmaf_rn(v[0], sc.is[0], rho0);
    // cx times ux, mxy and mxz (exact; zero for cx = 0 whatever they hold, infinities and NaN too)
    const float sx = (float)cx;
    const float uy = v[2], uz = v[3], mxx = v[4], myy = v[5], mzz = v[6], myz = v[9];
    const float sux = cx ? sx * v[1] : 0.f, smxy = cx ? sx * v[7] : 0.f, smxz = cx ? sx * v[8] : 0.f;
    const float t = __fadd_rn(__fadd_rn(mxx, myy), mzz);
    const float p0 = __fmaf_rn(-h15, t, 1.0f);
    const float a0 = cx ? __fmaf_rn(h45, mxx, p0) : p0;
    float e = a0;
    if constexpr (CY != 0 && CZ != 0) e = cx ? __fmaf_rn(h45, t, p0) : __fmaf_rn(h45, mzz, __fmaf_rn(h45, myy, p0));
    else if constexpr (CY != 0) e = __fmaf_rn(h45, myy, a0);
    else if constexpr (CZ != 0) e = __fmaf_rn(h45, mzz, a0);
    const float r = __fmul_rn(rho, kW2), q = __fmul_rn(h3, r), n = __fmul_rn(h9, r);
    float f = __fmul_rn(r, e);
    if constexpr (CY != 0 || CZ != 0) {
        float c = CY == 0 ? 0.f : (CY > 0 ? smxy : -smxy);
        if constexpr (CZ != 0) c = CY == 0 ? (CZ > 0 ? smxz : -smxz) : __fadd_rn(c, CZ > 0 ? smxz : -smxz);
        if constexpr (CY * CZ != 0) c = CY * CZ > 0 ? __fadd_rn(c, myz) : __fsub_rn(c, myz);
        f = __fmaf_rn(n, c, f);
    }
    float s = sux;
    if constexpr (CY != 0) s = CY > 0 ? __fadd_rn(s, uy) : __fsub_rn(s, uy);
    if constexpr (CZ != 0) s = CZ > 0 ? __fadd_rn(s, uz) : __fsub_rn(s, uz);
    f = __fmaf_rn(q, s, f);
    constexpr float w = (CY ? 1.0f : 4.0f) * (CZ ? 1.0f : 4.0f) * 0.25f;
    return f * (cx ? w : 4.0f * w);
}

// The populations of `mask` pulled by node (x, y, z) with this c_x, on the grid that wraps in every
// axis, into f[direction * stride].  Three lanes share a node, one per c_x: the three neighbours
// of a row mostly lie on one line.
template <typename S>
__device__ __forceinline__ void pull(const StepArgs &a, const S *__restrict__ src, uint32_t mask, int cx, int x, int y,
                                     int z, float *f, int stride) {
    constexpr int WPN = StorageLayout<S>::words;
    auto wrap = [](int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); };
    const int gx = wrap(x - cx, a.nx);
    const uint32_t *__restrict__ p = reinterpret_cast<const uint32_t *>(src) + (gx >> 5) * (WPN * kXBlock) + (gx & 31);
    const int64_t row = (int64_t)a.nxb * (WPN * kXBlock);
    // the loads of all nine rows go out together
    Raw<S> raw[9];
#pragma unroll
    for (int cz = -1; cz <= 1; ++cz) {
        const int64_t first = (int64_t)wrap(z - cz, a.nz) * a.ny;
#pragma unroll
        for (int cy = -1; cy <= 1; ++cy) {
            const int r = 3 * (cz + 1) + cy + 1;
            const int q = cx < 0 ? direction(-1, cy, cz) : (cx > 0 ? direction(1, cy, cz) : direction(0, cy, cz));
            if (mask >> q & 1u) load_raw_words<S>(p + (first + wrap(y - cy, a.ny)) * row, raw[r]);
            else raw[r] = Raw<S>{};
        }
    }
    auto put = [&](auto cyc, auto czc) {
        constexpr int cy = decltype(cyc)::value, cz = decltype(czc)::value;
        const int q = cx < 0 ? direction(-1, cy, cz) : (cx > 0 ? direction(1, cy, cz) : direction(0, cy, cz));
        float v[10];
        raw_values<S>(raw[3 * (cz + 1) + cy + 1], v);
        f[q * stride] = population<S, cy, cz>(v, cx, a.rho0, a.sc);
    };
    auto plane = [&](auto czc) {
        put(std::integral_constant<int, -1>{}, czc);
        put(std::integral_constant<int, 0>{}, czc);
        put(std::integral_constant<int, 1>{}, czc);
    };
    plane(std::integral_constant<int, -1>{});
    plane(std::integral_constant<int, 0>{});
    plane(std::integral_constant<int, 1>{});
}

// Populations that the closure of a listed node uses.
__device__ __forceinline__ uint32_t needed(const StepArgs &a, uint32_t w) {
    const uint32_t cls = w & NW_CLASS_MASK;
    if (cls == C_INNER || cls == C_OUTER) return a.wall[cls == C_INNER ? 0 : 1].in_mask[w >> NW_PAYLOAD_SHIFT];
    if (cls == C_BCFLUID_INNER || cls == C_BCFLUID_OUTER) return a.tag_in[(w >> NW_PAYLOAD_SHIFT) & 0xFFu];
    const uint32_t walls = class_walls(cls);
    if (walls == 0u || ((walls & 2u) && a.current_update)) return 0x7FFFFFFu;
    uint32_t m = 0u;
#pragma unroll
    for (int q = 0; q < 27; ++q) m |= known_dir(walls, q) ? 1u << q : 0u;
    return m;
}

// Closure of one listed node from its pulled populations `fl`.  Returns 0 when the node is
// not stored here (wall nodes: the wall kernel finishes them), 1 to store the collided moments
// `m`, 2 to store them and count the node in the fluid diagnostics.
template <typename S>
__device__ __forceinline__ int special_node(const StepArgs &a, int parity, bool force, uint32_t w, const float *fl,
                                            int x, int y, int z, int slot, int x0, int y0, Mom &m) {
    const uint32_t cls = w & NW_CLASS_MASK;
    const S *__restrict__ src = (const S *)a.m[parity];
    bool wall_node = false;
    bool fluid = true;
    const Mom prev = load_mom<S>(src, aos_at<S>(x, y, z, a.nxb, a.ny), a.rho0, a.sc);
    m = prev;  // nodes without a closure keep their pre-stream moments
    if (cls == C_INNER || cls == C_OUTER) {
        const int wi = cls == C_INNER ? 0 : 1;
        const uint32_t bi = w >> NW_PAYLOAD_SHIFT;
        incoming_rotated(a.wall[wi].nx[bi], a.wall[wi].ny[bi], a.wall[wi].in_mask[bi], fl, m);
        wall_node = true;
        fluid = false;
    } else if (cls == C_BCFLUID_INNER || cls == C_BCFLUID_OUTER) {
        const uint32_t tag = (w >> NW_PAYLOAD_SHIFT) & 0xFFu;
        Mom o = prev;
        if (bcfluid_closure(tag, a.tag_in[tag], fl, a.bcf_strong, a.omega, o)) m = o;
    } else if (cls == C_BCSOLID_INNER || cls == C_BCSOLID_OUTER) {
        const uint32_t tag = (w >> NW_PAYLOAD_SHIFT) & 0xFFu;
        Mom o = prev;
        if (bcsolid_closure(tag, fl, a.omega, o)) m = o;
    } else {
        PlanarCtx c;
        c.omega = a.omega;
        c.u_max = a.u_max;
        c.rho0 = a.rho0;
        c.convective = a.convective;
        c.self_prev = prev;
        c.west_prev = prev;
        if (class_walls(cls) & 2u) {
            if (a.current_update) {
                // NEUMANN_CURRENT_UPDATE (boundaries.cuh:96-161): post-stream rho, u of the
                // x-1 neighbour and of the node itself instead of their stored moments
                c.west_prev = pulled_rho_u<S>(a, src, x - 1, y, z);
                c.self_prev = rho_u_of(fl);
            } else {
                c.west_prev = load_mom<S>(src, aos_at<S>(x - 1, y, z, a.nxb, a.ny), a.rho0, a.sc);
            }
        }
        Mom o = prev;
        if (planar_closure(cls, fl, c, o)) m = o;
    }
    if ((w & NW_STENCIL) && slot >= 0) {
        float *e = a.side + side_index(slot, x, y, z, x0, y0, a.nz, TILE_X, a.tile_y) * 16;
        store_side(e, m.rho - a.rho0, m.ux, m.uy, m.uz, m.mxx, m.myy, m.mzz, m.mxy, m.mxz, m.myz);
    }
    if (wall_node) return 0;
    const bool bcf = force && slot >= 0 && (cls == C_BCFLUID_INNER || cls == C_BCFLUID_OUTER);
    double fin[4] = {0.0, 0.0, 0.0, 0.0};
    const uint32_t tag = (w >> NW_PAYLOAD_SHIFT) & 0xFFu;
    if (bcf) masked_momentum(a.tag_in[tag], m, fin);
    collide(m, a.omega);
    if (bcf) {
        double fo[4];
        masked_momentum(a.tag_out[tag], m, fo);
        float *e = a.side + side_index(slot, x, y, z, x0, y0, a.nz, TILE_X, a.tile_y) * 16;
        reinterpret_cast<float2 *>(e)[5] = make_float2((float)(fin[0] - fo[0]), (float)(fin[1] - fo[1]));
        reinterpret_cast<float2 *>(e)[6] = make_float2((float)(fin[2] - fo[2]), (float)(fin[3] - fo[3]));
    }
    return fluid ? 2 : 1;
}

// A warp takes ten nodes at a time: three lanes of each gather its populations into shared memory, then one lane
// per node applies its closure.  With three such rounds a warp the closure fills its lanes, but fewer warps hide
// the loads: annulus 77 us instead of 72 (67 now), a cylinder's 17 k nodes 18 instead of 15.
constexpr int kListWarps = 4, kListThreads = 32 * kListWarps, kListNodes = 10;

// BATCH: each block serves the case named by its entry in BatchArgs::list_blocks.
template <typename S, bool BATCH>
__global__ void __launch_bounds__(kListThreads)
    special_list_kernel(const StepArgs *__restrict__ ga, const BatchArgs *__restrict__ ba, int parity, double *force,
                        double *__restrict__ diag_part) {
    __shared__ float gathered[kListWarps][27][kListNodes + 1];
    int b0 = blockIdx.x, nblk = gridDim.x;
    if constexpr (BATCH) {
        const int4 m = ba->list_blocks[blockIdx.x];
        ga = ba->cases[m.x];
        b0 = blockIdx.x - m.y;
        nblk = m.z;
    }
    const StepArgs &a = *ga;
    // a sampled step: the wall kernel, launched after this one, adds into the slot
    if (!BATCH && force && blockIdx.x == 0 && threadIdx.x < 10) force[threadIdx.x] = 0.0;
    S *__restrict__ dst = (S *)a.m[parity ^ 1];
    const int n_all = a.n_list;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double dm = 0.0, de = 0.0;
    for (int first = (b0 * kListWarps + warp) * kListNodes; first < n_all; first += nblk * kListWarps * kListNodes) {
        if (const int j = lane / 3; lane < 3 * kListNodes && first + j < n_all) {
            const uint64_t p = a.list_xyz[first + j];
            pull<S>(a, (const S *)a.m[parity], needed(a, a.list_word[first + j]), lane % 3 - 1, (int)(p & 0x1FFFFFu),
                    (int)((p >> 21) & 0x1FFFFFu), (int)(p >> 42), &gathered[warp][0][j], kListNodes + 1);
        }
        __syncwarp();
        const int i = first + lane;
        if (lane < kListNodes && i < n_all) {
            const uint64_t p = a.list_xyz[i];
            const int x = (int)(p & 0x1FFFFFu), y = (int)((p >> 21) & 0x1FFFFFu), z = (int)(p >> 42);
            const uint32_t w = a.list_word[i];
            float f[27];
#pragma unroll
            for (int q = 0; q < 27; ++q) f[q] = gathered[warp][q][lane];
            const int tx = x / TILE_X, ty = y / a.tile_y;
            const int slot = a.tile_slot[ty * a.tiles_x + tx];
            Mom m;
            const int code = special_node<S>(a, parity, force != nullptr, w, f, x, y, z, slot, tx * TILE_X, ty * a.tile_y, m);
            if (code) {
                const int64_t ai = aos_at<S>(x, y, z, a.nxb, a.ny);
                if (kScaled<S> && a.sr_step)
                    store_mom_sr<S>(dst, ai, m, a.rho0, a.sc, sr_key(sr_step_seed(*a.sr_step), x, y, z, a.nx, a.ny));
                else
                    store_mom<S>(dst, ai, m, a.rho0, a.sc);
            }
            if (code == 2 && diag_part) {
                dm += (double)(m.rho - a.rho0);
                de += 0.5 * (double)(m.ux * m.ux + m.uy * m.uy + m.uz * m.uz);
            }
        }
        __syncwarp();
    }
    if (diag_part) {
        // fixed-order block reduction -> diag_part[blockIdx.x]
        __shared__ double red[2][kListThreads / 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            dm += __shfl_down_sync(0xffffffffu, dm, o);
            de += __shfl_down_sync(0xffffffffu, de, o);
        }
        if ((threadIdx.x & 31) == 0) {
            red[0][threadIdx.x >> 5] = dm;
            red[1][threadIdx.x >> 5] = de;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double s0 = 0.0, s1 = 0.0;
            for (int k = 0; k < kListThreads / 32; ++k) {
                s0 += red[0][k];
                s1 += red[1][k];
            }
            diag_part[2 * blockIdx.x + 0] = s0;
            diag_part[2 * blockIdx.x + 1] = s1;
        }
    }
}

}  // namespace

int special_list_blocks(int n_list) {
    const int b = (n_list + kListWarps * kListNodes - 1) / (kListWarps * kListNodes);
    return b < 1 ? 1 : (b > 4096 ? 4096 : b);
}

cudaError_t launch_special_list(const StepLaunch &l, int storage, int n_blocks, double *diag_part, cudaStream_t s) {
    double *const f = l.force;
    switch (storage) {
        case MRLBM_STORAGE_F32:
            special_list_kernel<float, false><<<n_blocks, kListThreads, 0, s>>>(l.ga, nullptr, l.parity, f, diag_part);
            break;
        case MRLBM_STORAGE_F16:
            special_list_kernel<__half, false><<<n_blocks, kListThreads, 0, s>>>(l.ga, nullptr, l.parity, f, diag_part);
            break;
        case MRLBM_STORAGE_BF16:
            special_list_kernel<__nv_bfloat16, false>
                <<<n_blocks, kListThreads, 0, s>>>(l.ga, nullptr, l.parity, f, diag_part);
            break;
        case MRLBM_STORAGE_F16_U32:
            special_list_kernel<HybridWord, false>
                <<<n_blocks, kListThreads, 0, s>>>(l.ga, nullptr, l.parity, f, diag_part);
            break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_special_list_batch(const BatchArgs *ba, int parity, int force, int storage, int n_blocks,
                                      cudaStream_t s) {
    if (n_blocks <= 0) return cudaSuccess;
    // any non-null pointer makes it a sampled step (the batch has zeroed its cases' slots)
    double *const f = force ? reinterpret_cast<double *>(1) : nullptr;
    switch (storage) {
        case MRLBM_STORAGE_F32:
            special_list_kernel<float, true><<<n_blocks, kListThreads, 0, s>>>(nullptr, ba, parity, f, nullptr);
            break;
        case MRLBM_STORAGE_F16:
            special_list_kernel<__half, true><<<n_blocks, kListThreads, 0, s>>>(nullptr, ba, parity, f, nullptr);
            break;
        case MRLBM_STORAGE_BF16:
            special_list_kernel<__nv_bfloat16, true>
                <<<n_blocks, kListThreads, 0, s>>>(nullptr, ba, parity, f, nullptr);
            break;
        case MRLBM_STORAGE_F16_U32:
            special_list_kernel<HybridWord, true>
                <<<n_blocks, kListThreads, 0, s>>>(nullptr, ba, parity, f, nullptr);
            break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace mrlbm
