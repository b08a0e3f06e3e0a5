// sm_100a kernels of the SCMF engine.
//
//   k_init_coords   random-walk chains (device_function.cu:140-207)
//   k_sweep_warp    one MC sweep on warp tiles, of linear chains and other bond
//                   graphs of up to six bonds a bead (scmf_sweep.cuh): odd/even or
//                   colour by colour, smart-MC trials (device_function.cu:444-454,
//                   509-799), moving one cell count for each accepted move that
//                   leaves its cell, so counts stay the grid of the positions
//                   (device_function.cu:471-508)
//   k_sweep_pairs   the same in registers, where no trial is screened
//   k_run           many whole sweeps, where the positions fit on the chip
//   k_sweep         a sweep of what these do not take (longer chains, more bonds)
//   k_grid          counts of the current positions from scratch
//   k_field<fused>  counts -> omega (SCMF0, device_function.cu:373-412) with the
//                   field-energy reduction; in the fused step the block that
//                   finishes a system's last tile closes the sweep (step,
//                   statistics, averaging sample)
//   k_close, k_bond_energy, k_observables, k_validate_*, transposes: the
//                   reductions and checks around the step
//
// Built with --fmad=false -prec-div=true -prec-sqrt=true: positions and counts
// are bit-identical to the CPU oracle, whatever the tiling or launch shape.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "scmf.h"

#include "scmf_internal.h"
#include "scmf_math.cuh"
#include "scmf_normal_table.h"
#include "scmf_screen_table.h"

namespace scmf {

// The inverse normal CDF table of normal_of, read-only in global memory.
__device__ __align__(16) const float g_normal_tab[SCMF_NORMAL_SEGS * 4] = {SCMF_NORMAL_TABLE_DATA};

// The screen's piecewise-linear table (scmf_sweep.cuh).
__device__ __align__(16) const float g_screen_tab[SCMF_SCREEN_SEGS * 2] = {SCMF_SCREEN_TABLE_DATA};

__device__ __forceinline__ const float2* screen_table() { return reinterpret_cast<const float2*>(g_screen_tab); }
__device__ __forceinline__ const float4* normal_table() { return reinterpret_cast<const float4*>(g_normal_tab); }

// i / n via a multiply-high by magic = ceil(2^32 / n) (exact while i * n < 2^32).
__device__ __forceinline__ uint32_t div_magic(uint32_t i, uint32_t magic, int n) {
    return n == 1 ? i : __umulhi(i, magic);
}

// ------------------------------------------------------------------ init
__global__ void k_init_coords(SysDev* __restrict__ S, const ArchDev* __restrict__ archs, int n_arch,
                              int n_chains) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n_chains) return;
    int a = 0;
    while (a + 1 < n_arch && g >= archs[a + 1].chain_base) ++a;
    const ArchDev& A = archs[a];
    const int L = A.length;
    const int64_t b0 = A.bead_base + (int64_t)(g - A.chain_base) * L;
    const uint32_t gid = (uint32_t)(A.rng_base + (g - A.chain_base));  // the chain's random-stream id
    float* X = S->x + b0;
    float* Y = S->y + b0;
    float* Z = S->z + b0;
    const uint32_t k0 = S->seed_lo, k1 = S->seed_hi;
    uint32_t placed[kMaxLength / 32];
    for (int i = 0; i < (L + 31) / 32; ++i) placed[i] = 0u;
    for (int i = 0; i < L; ++i) {
        X[i] = 0.0f;
        Y[i] = 0.0f;
        Z[i] = 0.0f;
    }
    uint4 w = philox4x32_10(make_uint4(gid, 0u, kInitStep, 0u), k0, k1);
    X[0] = u01(w.x) * S->lx;
    Y[0] = u01(w.y) * S->ly;
    Z[0] = u01(w.z) * S->lz;
    placed[0] = 1u;
    for (int i = 0; i < L; ++i) {
        const BeadInfo bi = A.beads[i];
        for (int d = 0; d < bi.deg; ++d) {
            const int j = bi.nbr[d];
            if (placed[j >> 5] & (1u << (j & 31))) continue;
            float n0, n1, n2;
            normals3(philox4x32_10(make_uint4(gid, (uint32_t)j, kInitStep, 1u), k0, k1), normal_table(), n0, n1, n2);
            X[j] = X[i] + A.init_sigma * n0;
            Y[j] = Y[i] + A.init_sigma * n1;
            Z[j] = Z[i] + A.init_sigma * n2;
            placed[j >> 5] |= 1u << (j & 31);
        }
    }
}

// ------------------------------------------------------------------ sweep
struct MoveConsts {
    float k, k2, A, R, inv_dx, inv_dy, inv_dz;
    float span;  // SysDev::omega_span of the system (early rejection)
    int nx, ny, nz;
    bool pow2;   // every axis a power of two
    bool small;  // every axis of 2 to 256 cells (fold_magic)
};

__device__ __forceinline__ bool is_pow2(int n) { return (n & (n - 1)) == 0; }

__device__ __forceinline__ void load_fold(MoveConsts& c, const SysDev* S) {
    c.span = S->omega_span;
    c.nx = S->nx; c.ny = S->ny; c.nz = S->nz;
    c.pow2 = is_pow2(c.nx) && is_pow2(c.ny) && is_pow2(c.nz);
    c.small = c.nx >= 2 && c.ny >= 2 && c.nz >= 2 && c.nx <= 256 && c.ny <= 256 && c.nz <= 256;
}

// Offsets and magic multipliers of fold_magic for n = 0 .. 256 (filled once
// per device by configure_kernels).  Every lane of a warp reads the entry of
// the same n, which the constant cache broadcasts.
__constant__ int2 c_fold[257];

// Cell index of a position; the system's grid picks the fold.
__device__ __forceinline__ int cell_of(const MoveConsts& c, float x, float y, float z) {
    int ix, iy, iz;
    if (c.pow2) {
        ix = fold_pow2(x, c.inv_dx, c.nx - 1);
        iy = fold_pow2(y, c.inv_dy, c.ny - 1);
        iz = fold_pow2(z, c.inv_dz, c.nz - 1);
    } else if (c.small) {
        const int2 fx = c_fold[c.nx], fy = c_fold[c.ny], fz = c_fold[c.nz];
        ix = fold_magic(x, c.inv_dx, c.nx, fx.x, (uint32_t)fx.y);
        iy = fold_magic(y, c.inv_dy, c.ny, fy.x, (uint32_t)fy.y);
        iz = fold_magic(z, c.inv_dz, c.nz, fz.x, (uint32_t)fz.y);
    } else {
        ix = fold(x, c.inv_dx, c.nx);
        iy = fold(y, c.inv_dy, c.ny);
        iz = fold(z, c.inv_dz, c.nz);
    }
    return ix + c.nx * (iy + c.ny * iz);
}


// Bond force f = 2k sum_j (q_j - p), one neighbour at a time in ascending
// bead order (fma per neighbour, as the oracle).
__device__ __forceinline__ void add_bond(float k2, float x, float y, float z, float qx, float qy, float qz, float& fx,
                                         float& fy, float& fz) {
    fx = __fmaf_rn(__fsub_rn(qx, x), k2, fx);
    fy = __fmaf_rn(__fsub_rn(qy, y), k2, fy);
    fz = __fmaf_rn(__fsub_rn(qz, z), k2, fz);
}

// Rejection before the omega reads.  Every field step publishes span >= the
// largest omega_t[a] - omega_t[b] (SysDev::omega_span), so, rounding being
// monotone, fl(w_new - w_old) >= -span and dE = fl(fl(w_new - w_old) + deb) >=
// fl(deb - span) =: lb.  A trial with -lb <= log_lower(u) <= log_f(u) has
// dE > 0 and log_f(u) >= -dE: the Metropolis test below rejects it whatever
// omega holds (and a NaN bound or energy rejects, as the test does).  At the
// benchmark acceptance (~0.5 %) about 2 % of trials pass this bound, so about
// half of the warps skip the cell folds, the two gathers and their L2 round
// trip altogether; the outcome of every trial is the oracle's.
__device__ __forceinline__ bool maybe_accepted(float deb, float span, float lf) {
    return -__fsub_rn(deb, span) > lf;
}

// The trial of a bead at (x,y,z) with bond force f.  With d = A f + R xi the
// displacement, the reference's bonded energy change plus smart-MC correction
// equals (A c / 4)(c |d|^2 - 2 f.d), c = 2k deg (the force at p + d is
// f - c d).  Same FP32 expression (explicit fma) as the oracle's move_bead().
// Returns whether the move is accepted; (px,py,pz) is the proposed position
// and cell_old / cell_new the cells of the old and proposed positions.
__device__ __forceinline__ bool trial_f(const MoveConsts& c, float x, float y, float z, float fx, float fy, float fz,
                                        float cc, float ac4, float n0, float n1, float n2, uint32_t aw,
                                        const float* __restrict__ w_t, float& px, float& py, float& pz, int& cell_old,
                                        int& cell_new) {
    const float A = c.A, R = c.R;
    const float dx = __fmaf_rn(A, fx, __fmul_rn(R, n0));
    const float dy = __fmaf_rn(A, fy, __fmul_rn(R, n1));
    const float dz = __fmaf_rn(A, fz, __fmul_rn(R, n2));
    px = __fadd_rn(x, dx);
    py = __fadd_rn(y, dy);
    pz = __fadd_rn(z, dz);
    const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
    const float fd = __fmaf_rn(fx, dx, __fmaf_rn(fy, dy, __fmul_rn(fz, dz)));
    const float deb = __fmul_rn(ac4, __fmaf_rn(cc, d2, __fmul_rn(-2.0f, fd)));
    // Trials that the omega span already rejects skip the folds and gathers
    // (maybe_accepted; same outcome).  Otherwise: log(u) >= -23 ln2 > -17 for
    // every u the generator yields, so dE >= 17 rejects without the logarithm;
    // below that, log_f(u) >= log_lower(u) for every such u, so
    // -dE <= log_lower(u) rejects without it too (same outcome).
    bool acc = false;
    int c_old = 0, c_new = 0;
    if (maybe_accepted(deb, c.span, log_lower(u01(aw)))) {
        c_old = cell_of(c, x, y, z);
        c_new = cell_of(c, px, py, pz);
        const float dE = __fadd_rn(__fsub_rn(__ldg(w_t + c_new), __ldg(w_t + c_old)), deb);
        if (dE < 0.0f)
            acc = true;
        else if (dE < 17.0f)
            acc = -dE > log_lower(u01(aw)) && log_f(u01(aw)) < -dE;  // u recomputed: no register held across
    }
    cell_old = c_old;
    cell_new = c_new;
    return acc;
}

// One smart-MC trial (device_function.cu:637-717, 562-588, 444-454) of a bead
// at (x,y,z) with deg bonded neighbours q[0..deg) in ascending bead order.
template <int MAXDEG>
__device__ __forceinline__ bool trial(const MoveConsts& c, float x, float y, float z, const float* qx,
                                      const float* qy, const float* qz, int deg, float cc, float ac4, float n0,
                                      float n1, float n2, uint32_t aw, const float* __restrict__ w_t, float& px,
                                      float& py, float& pz, int& cell_old, int& cell_new) {
    float fx = 0.0f, fy = 0.0f, fz = 0.0f;
#pragma unroll
    for (int d = 0; d < MAXDEG; ++d)
        if (d < deg) add_bond(c.k2, x, y, z, qx[d], qy[d], qz[d], fx, fy, fz);
    return trial_f(c, x, y, z, fx, fy, fz, cc, ac4, n0, n1, n2, aw, w_t, px, py, pz, cell_old, cell_new);
}

// Counts are kept as the grid of the current positions: a fused sweep moves
// one count from the old to the new cell of every accepted move that leaves
// its cell (typ = type * n_cells), instead of regridding every bead.
__device__ __forceinline__ void count_move(uint32_t* cnt, bool c16, int64_t typ, int c_old, int c_new) {
    const int64_t io = typ + c_old, in = typ + c_new;
    if (c16) {
        atomicSub(cnt + (io >> 1), 1u << ((io & 1) * 16));  // the cell holds this bead: no borrow
        atomicAdd(cnt + (in >> 1), 1u << ((in & 1) * 16));
    } else {
        atomicSub(cnt + io, 1u);
        atomicAdd(cnt + in, 1u);
    }
}

// KEYS (KeyMode): kKeysBoth when every system of the launch has the seed whose
// Philox round keys are in `keys` (a kernel parameter); kKeysHigh when they
// share its upper 32 bits, so that only the first key word is read from the
// tile's SysDev and advanced round by round; kKeysNone: both are.
template <int KEYS>
__device__ __forceinline__ uint4 philox_block(uint4 ctr, uint32_t k0, uint32_t k1, const PhiloxKeys& keys) {
    if (KEYS == kKeysBoth) return philox4x32_10(ctr, keys);
    if (KEYS == kKeysHigh) return philox4x32_10(ctr, k0, keys);
    return philox4x32_10(ctr, k0, k1);
}

// Philox block and normals of bead b of chain gc; returns its Metropolis word.
template <int KEYS>
__device__ __forceinline__ uint32_t bead_normals(uint32_t gc, int b, uint32_t step, uint32_t k0, uint32_t k1,
                                                 const PhiloxKeys& keys, float& n0, float& n1, float& n2) {
    const uint4 w = philox_block<KEYS>(make_uint4(gc, (uint32_t)b, step, 0u), k0, k1, keys);
    normals3(w, normal_table(), n0, n1, n2);
    return accept_word(w);
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

size_t sweep_smem_bytes(int max_tile_beads, int max_length) {
    size_t b = (size_t)max_tile_beads * 3 * sizeof(float);
    b = (b + 15) & ~(size_t)15;
    b += (size_t)max_length * sizeof(BeadInfo);
    b = (b + 15) & ~(size_t)15;
    b += (size_t)max_length * sizeof(uint16_t);
    return (b + 15) & ~(size_t)15;
}

// One MC sweep over tiles of whole chains staged in shared memory: of plans that
// the kernels of warp tiles do not take (a bead of more than six bonds, a chain longer than a
// warp's tile, 2^31 cells times types), every trial made exactly.
//   MODE kMoveOnly / kMoveGrid: moves; moves keeping counts[cur] the grid of
//   the positions (accepted moves that change cell move a count).
//   Two 256-thread CTAs per SM leave it 128 registers and no spill (at 64 it
//   spilled ~400 B per thread and moved combs 12 % slower).
template <int MODE, int KEYS>
__global__ void __launch_bounds__(256, 2) k_sweep(const MoveTile* __restrict__ tiles, int n_tiles,
                                                   int max_tile_beads, int max_length, const PhiloxKeys keys) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* sx = reinterpret_cast<float*>(smem_raw);
    float* sy = sx + max_tile_beads;
    float* sz = sy + max_tile_beads;
    size_t off = ((size_t)max_tile_beads * 3 * sizeof(float) + 15) & ~(size_t)15;
    BeadInfo* sinfo = reinterpret_cast<BeadInfo*>(smem_raw + off);
    off = (off + (size_t)max_length * sizeof(BeadInfo) + 15) & ~(size_t)15;
    uint16_t* scol = reinterpret_cast<uint16_t*>(smem_raw + off);
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
    for (int ti = blockIdx.x; ti < n_tiles; ti += gridDim.x) {
        const MoveTile t = tiles[ti];
        SysDev* S = t.sys;
        if (S->step >= S->stop_step) continue;  // block-uniform
        const ArchDev* Ap = t.arch;
        const int L = Ap->length;
        const int nb = t.n_chains * L;
        if (nb > max_tile_beads || L > max_length) {
            if (tid == 0) atomicOr(&S->error_word, kErrorSize);
            continue;
        }
        MoveConsts c;
        c.k = S->k; c.k2 = S->k2; c.A = S->A; c.R = S->R;
        c.inv_dx = S->inv_dx; c.inv_dy = S->inv_dy; c.inv_dz = S->inv_dz;
        load_fold(c, S);
        for (int i = tid; i < L; i += T) {
            sinfo[i] = Ap->beads[i];
            scol[i] = Ap->color_beads[i];
        }
        float* gx = S->x + t.bead0;
        float* gy = S->y + t.bead0;
        float* gz = S->z + t.bead0;
        const bool vec = ((t.bead0 & 3) == 0) && ((nb & 3) == 0);
        if (vec) {
            const float4* vx = reinterpret_cast<const float4*>(gx);
            const float4* vy = reinterpret_cast<const float4*>(gy);
            const float4* vz = reinterpret_cast<const float4*>(gz);
            for (int i = tid; i < (nb >> 2); i += T) {
                const float4 a = __ldcs(vx + i), b = __ldcs(vy + i), d = __ldcs(vz + i);
                reinterpret_cast<float4*>(sx)[i] = a;
                reinterpret_cast<float4*>(sy)[i] = b;
                reinterpret_cast<float4*>(sz)[i] = d;
            }
        } else {
            for (int i = tid; i < nb; i += T) {
                sx[i] = gx[i];
                sy[i] = gy[i];
                sz[i] = gz[i];
            }
        }
        __syncthreads();

        {
            const uint32_t step = S->step + 1u;
            const uint32_t k0 = S->seed_lo, k1 = S->seed_hi;
            const uint32_t* __restrict__ cid = S->chain_id + t.chain0;
            const float* __restrict__ omega = S->omega;
            const int64_t NC = S->n_cells;
            const float cc2 = S->cdeg[2], ac42 = S->ac4deg[2];
            uint32_t* cnt = S->counts[S->cur];
            const bool c16 = S->count16 != 0;
            unsigned nacc = 0;
            for (int col = 0; col < Ap->n_colors; ++col) {
                const int ncol = Ap->color_off[col + 1] - Ap->color_off[col];
                const uint32_t mg = Ap->color_magic[col];
                const int items = t.n_chains * ncol;
                for (int j = tid; j < items; j += T) {
                    const int cl = (int)div_magic((uint32_t)j, mg, ncol);
                    const int base = cl * L;
                    float qx[kMaxDeg], qy[kMaxDeg], qz[kMaxDeg];
                    int b, deg, type;
                    b = scol[Ap->color_off[col] + (j - cl * ncol)];
                    const BeadInfo bi = sinfo[b];
                    type = bi.type;
                    deg = bi.deg;
#pragma unroll
                    for (int d = 0; d < kMaxDeg; ++d) {
                        if (d < deg) {
                            const int q = base + bi.nbr[d];
                            qx[d] = sx[q];
                            qy[d] = sy[q];
                            qz[d] = sz[q];
                        }
                    }
                    float n0, n1, n2;
                    const uint32_t aw = bead_normals<KEYS>(__ldg(cid + cl), b, step, k0, k1, keys, n0, n1, n2);
                    float px, py, pz;
                    int c_old, c_new;
                    const bool acc = trial<kMaxDeg>(c, sx[base + b], sy[base + b], sz[base + b], qx, qy,
                                                                 qz, deg, deg == 2 ? cc2 : S->cdeg[deg],
                                                                 deg == 2 ? ac42 : S->ac4deg[deg], n0, n1, n2, aw,
                                                                 omega + (int64_t)type * NC, px, py, pz, c_old, c_new);
                    if (acc) {
                        sx[base + b] = px;
                        sy[base + b] = py;
                        sz[base + b] = pz;
                    }
                    nacc += acc ? 1u : 0u;
                    if (MODE == kMoveGrid && acc && c_new != c_old) count_move(cnt, c16, (int64_t)type * NC, c_old, c_new);
                }
                __syncthreads();
            }
            nacc = warp_sum(nacc);
            if (lane == 0 && nacc) atomicAdd(&S->slot_acc[(ti * kMaxWarps + warp) % kSlots], (unsigned long long)nacc);
        }

        {
            if (vec) {
                float4* vx = reinterpret_cast<float4*>(gx);
                float4* vy = reinterpret_cast<float4*>(gy);
                float4* vz = reinterpret_cast<float4*>(gz);
                for (int i = tid; i < (nb >> 2); i += T) {
                    __stcs(vx + i, reinterpret_cast<const float4*>(sx)[i]);
                    __stcs(vy + i, reinterpret_cast<const float4*>(sy)[i]);
                    __stcs(vz + i, reinterpret_cast<const float4*>(sz)[i]);
                }
            } else {
                for (int i = tid; i < nb; i += T) {
                    gx[i] = sx[i];
                    gy[i] = sy[i];
                    gz[i] = sz[i];
                }
            }
        }
        __syncthreads();
    }
}

// Counts of the current positions added into counts[cur] (a cleared buffer),
// over the tiles of the launch (device_function.cu:471-508).
__global__ void __launch_bounds__(256) k_grid(const MoveTile* __restrict__ tiles, int n_tiles) {
    for (int ti = blockIdx.x; ti < n_tiles; ti += gridDim.x) {
        const MoveTile t = tiles[ti];
        SysDev* S = t.sys;
        const ArchDev* Ap = t.arch;
        const int L = Ap->length;
        const int nb = t.n_chains * L;
        MoveConsts c;
        c.inv_dx = S->inv_dx; c.inv_dy = S->inv_dy; c.inv_dz = S->inv_dz;
        load_fold(c, S);
        const float* X = S->x + t.bead0;
        const float* Y = S->y + t.bead0;
        const float* Z = S->z + t.bead0;
        uint32_t* cnt = S->counts[S->cur];
        const int64_t NC = S->n_cells;
        const bool c16 = S->count16 != 0;
        const uint8_t* __restrict__ types = Ap->types;
        const uint32_t len_magic = Ap->len_magic;
        for (int i = threadIdx.x; i < nb; i += blockDim.x) {
            const int b = i - (int)div_magic((uint32_t)i, len_magic, L) * L;
            const int64_t idx = (int64_t)__ldg(types + b) * NC + cell_of(c, X[i], Y[i], Z[i]);
            if (c16)
                atomicAdd(cnt + (idx >> 1), 1u << ((idx & 1) * 16));
            else
                atomicAdd(cnt + idx, 1u);
        }
    }
}


// ------------------------------------------------------------------ field

// omega of one cell from its counts (NT = 0: runtime type count, up to
// kMaxTypes).  Expression order matches the oracle's field_update():
// phi_S = n_S * scale, tot = sum_S phi_S (S ascending), then
// SCMF0: w_T = (tot - 1) cf_TT + sum_{S != T} cf_TS (phi_T - phi_S)
// literal: w_T = (tot - 1) cf_TT + sum_{S != T} cf_TS phi_S.
// Returns the cell's field energy, or 0 without `energy` (its conversions to FP64
// take longer than all the rest).
template <int NT>
__device__ __forceinline__ double omega_of_cell(int nt, const uint32_t* cnt, float scale, bool lit, bool upd, float* w,
                                                const float* cf, bool energy = true) {
    constexpr int M = NT > 0 ? NT : kMaxTypes;
    float phi[M];
    float tot = 0.0f;
#pragma unroll
    for (int u = 0; u < M; ++u) {
        if (u < nt) {
            phi[u] = (float)cnt[u] * scale;
            tot = tot + phi[u];
        }
    }
    double ef = 0.0;
#pragma unroll
    for (int t = 0; t < M; ++t) {
        if (t < nt) {
            if (upd) {
                float v = (tot - 1.0f) * cf[t + nt * t];
#pragma unroll
                for (int u = 0; u < M; ++u) {
                    if (u < nt && u != t) {
                        if (!lit)
                            v = v + cf[t + nt * u] * (phi[t] - phi[u]);
                        else
                            v = v + cf[t + nt * u] * phi[u];
                    }
                }
                w[t] = v;
            }
            if (energy) ef += (double)w[t] * (double)cnt[t];
        }
    }
    return ef;
}

// Scalar path: one cell (any count width, any alignment).  FROM_L2: counts and
// omega change in the course of the launch, so they are not read through L1.
template <int NT, bool FROM_L2>
__device__ __forceinline__ double field_cell(int n, int64_t cell, int64_t NC, float scale, bool lit, bool upd,
                                             bool c16, const uint32_t* src32, float* W, const float* cf,
                                             unsigned long long* avg, float& wmax, float& wmin,
                                             bool energy = true) {
    constexpr int M = NT > 0 ? NT : kMaxTypes;
    const int nt = NT > 0 ? NT : n;
    const uint16_t* src16 = reinterpret_cast<const uint16_t*>(src32);
    uint32_t cnt[M];
    float w[M];
#pragma unroll
    for (int u = 0; u < M; ++u) {
        if (u < nt) {
            const int64_t i = u * NC + cell;
            if (FROM_L2) {
                cnt[u] = c16 ? (uint32_t)__ldcg(src16 + i) : __ldcg(src32 + i);
                if (!upd) w[u] = __ldcg(W + i);
            } else {
                cnt[u] = c16 ? (uint32_t)src16[i] : src32[i];
                if (!upd) w[u] = W[i];
            }
            if (avg) avg[u * NC + cell] += cnt[u];
        }
    }
    const double ef = omega_of_cell<NT>(nt, cnt, scale, lit, upd, w, cf, energy);
#pragma unroll
    for (int t = 0; t < M; ++t) {
        if (t < nt && upd) W[t * NC + cell] = w[t];
        if (t < nt) {
            wmax = fmaxf(wmax, w[t]);  // fmaxf / fminf skip NaN
            wmin = fminf(wmin, w[t]);
        }
    }
    return ef;
}

// Vector path: four consecutive cells with 16-byte loads and stores (32-bit
// counts, n_cells and the tile start multiples of 4).
template <int NT, bool FROM_L2>
__device__ __forceinline__ double field_cells4(int64_t cell, int64_t NC, float scale, bool lit, bool upd,
                                               const uint32_t* src32, float* W, const float* cf,
                                               unsigned long long* avg, float& wmax, float& wmin,
                                               bool energy = true) {
    uint4 cv[NT];
    float4 wv[NT];
#pragma unroll
    for (int u = 0; u < NT; ++u) {
        const uint4* const c = reinterpret_cast<const uint4*>(src32 + u * NC + cell);
        const float4* const w = reinterpret_cast<const float4*>(W + u * NC + cell);
        cv[u] = FROM_L2 ? __ldcg(c) : *c;
        if (!upd) wv[u] = FROM_L2 ? __ldcg(w) : *w;
    }
    if (avg) {
#pragma unroll
        for (int u = 0; u < NT; ++u) {
            ulonglong2* a = reinterpret_cast<ulonglong2*>(avg + u * NC + cell);
            ulonglong2 lo = a[0], hi = a[1];
            lo.x += cv[u].x; lo.y += cv[u].y;
            hi.x += cv[u].z; hi.y += cv[u].w;
            a[0] = lo;
            a[1] = hi;
        }
    }
    double ef = 0.0;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        uint32_t cnt[NT];
        float w[NT];
#pragma unroll
        for (int u = 0; u < NT; ++u) {
            cnt[u] = l == 0 ? cv[u].x : l == 1 ? cv[u].y : l == 2 ? cv[u].z : cv[u].w;
            w[u] = l == 0 ? wv[u].x : l == 1 ? wv[u].y : l == 2 ? wv[u].z : wv[u].w;
        }
        ef += omega_of_cell<NT>(NT, cnt, scale, lit, upd, w, cf, energy);
#pragma unroll
        for (int u = 0; u < NT; ++u) {
            wmax = fmaxf(wmax, w[u]);
            wmin = fminf(wmin, w[u]);
            if (l == 0) wv[u].x = w[u];
            else if (l == 1) wv[u].y = w[u];
            else if (l == 2) wv[u].z = w[u];
            else wv[u].w = w[u];
        }
    }
#pragma unroll
    for (int u = 0; u < NT; ++u) {
        if (upd) *reinterpret_cast<float4*>(W + u * NC + cell) = wv[u];
    }
    return ef;
}

// Order-preserving integer key of a non-NaN float (for atomicMax / atomicMin)
// and its inverse.
__device__ __forceinline__ uint32_t ord_key(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord_val(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

}  // namespace scmf

#include "scmf_sweep.cuh"

namespace scmf {

// Closes one system after a launch (one block): sums the accept slots and the
// energy partials part[0 .. count) in an order fixed by the block size, and
// thread 0 publishes the statistics and, for a full sweep, advances the step
// and makes the new counts current.  Partials written by other blocks of the
// same launch are read through L2.
__device__ void close_system(SysDev* S, const double* part, int count, int mode, unsigned long long* s_a,
                             double* s_f) {
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long a = 0;
    double f = 0.0;
    if ((mode & kCloseMove) && tid < kSlots) {
        a = __ldcg(&S->slot_acc[tid]);
        S->slot_acc[tid] = 0ull;
    }
    if (mode & (kCloseField | kCloseBond))
        for (int i = tid; i < count; i += T) f += __ldcg(part + i);
    a = warp_sum(a);
    f = warp_sum(f);
    if (lane == 0) {
        s_a[warp] = a;
        s_f[warp] = f;
    }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < (T + 31) / 32; ++w) {
            a += s_a[w];
            f += s_f[w];
        }
        if (mode & kCloseMove) {
            S->last_accepts = a;
            S->total_accepts += a;
            S->total_moves += (unsigned long long)S->n_beads;
        }
        if (mode & kCloseField) S->e_field = f;
        if (mode & kCloseBond) {
            S->e_bond = f;
            S->e_bond_step = S->step + 1u;
        }
        if ((mode & kCloseAverage) && S->avg && S->avg_every && ((S->step + 1u) % S->avg_every) == 0u)
            S->avg_samples += 1ull;
        if (mode & kCloseAdvance) S->step += 1u;
    }
    __syncthreads();
}

template <bool FUSED, int NT>
__global__ void __launch_bounds__(256) k_field(const FieldTile* __restrict__ tiles, int n_tiles, int force_update,
                                                double* __restrict__ ef_part, int close_mode) {
    __shared__ double s_ef[32];
    __shared__ float s_mx[32], s_mn[32];
    __shared__ unsigned long long s_acc[32];
    __shared__ float cf[kMaxTypes * kMaxTypes];
    __shared__ int s_last;
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
    for (int ti = blockIdx.x; ti < n_tiles; ti += gridDim.x) {
        const FieldTile t = tiles[ti];
        SysDev* S = t.sys;
        for (int i = tid; i < kMaxTypes * kMaxTypes; i += T) cf[i] = S->cf[i];
        const int n = S->n_types, rule = S->field_rule;
        const int64_t NC = S->n_cells;
        const float scale = S->scale;
        const bool lit = S->hamiltonian == 1;
        const bool c16 = S->count16 != 0;
        const uint32_t* src32 = S->field_counts ? S->field_counts : S->counts[S->cur];
        float* W = S->omega;
        unsigned long long* avg = FUSED && S->avg_every ? S->avg : nullptr;
        const uint32_t avg_every = S->avg_every, stop = S->stop_step;
        // all that a sweep leaves as it is has been read; a launch beside the move kernel's
        // last blocks (LaunchShape::chained) waits for the rest of it here
        if (FUSED && ti == (int)blockIdx.x) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        }
        __syncthreads();
        const uint32_t sweep = S->step + 1u;
        if (FUSED && sweep > stop) continue;  // block-uniform: the system's sweeps are done
        const bool upd = force_update || rule == 1 || (sweep % 10u) != 0u;
        // the fused sweep samples the time-averaged density at every avg_every-th sweep
        if (avg && sweep % avg_every != 0u) avg = nullptr;
        // the energy of a sweep that another one follows in the same call is not asked for
        const int mode = FUSED && sweep == stop ? close_mode | kCloseField : close_mode;
        const bool energy = !FUSED || (mode & kCloseField) != 0;
        double ef = 0.0;
        float wmax = -INFINITY, wmin = INFINITY;  // omega of the tile's cells (new or kept)
        const int64_t end = t.cell0 + t.n_cells;
        if (NT > 0 && !c16 && (NC & 3) == 0 && (t.cell0 & 3) == 0 && (t.n_cells & 3) == 0) {
            for (int64_t cell = t.cell0 + 4 * tid; cell < end; cell += 4 * T)
                ef += field_cells4<(NT > 0 ? NT : 1), false>(cell, NC, scale, lit, upd, src32, W, cf, avg, wmax, wmin, energy);
        } else {
            for (int64_t cell = t.cell0 + tid; cell < end; cell += T)
                ef += field_cell<NT, false>(n, cell, NC, scale, lit, upd, c16, src32, W, cf, avg, wmax, wmin, energy);
        }
        if (energy) ef = warp_sum(ef);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            wmax = fmaxf(wmax, __shfl_xor_sync(0xffffffffu, wmax, o));
            wmin = fminf(wmin, __shfl_xor_sync(0xffffffffu, wmin, o));
        }
        if (lane == 0) {
            s_ef[warp] = ef;
            s_mx[warp] = wmax;
            s_mn[warp] = wmin;
        }
        __syncthreads();
        if (tid == 0) {
            double e = 0.0;
            for (int w = 0; w < (T + 31) / 32; ++w) {
                if (energy) e += s_ef[w];
                wmax = fmaxf(wmax, s_mx[w]);
                wmin = fminf(wmin, s_mn[w]);
            }
            if (energy) ef_part[ti] = e;
            if (wmax >= wmin) {  // the tile held a non-NaN omega
                atomicMax(&S->om_max_key, ord_key(wmax));
                atomicMin(&S->om_min_key, ord_key(wmin));
            }
            if (close_mode) {
                // publish the partial, then count the tile; the block that
                // finishes a system's last tile closes it (no waiting)
                __threadfence();
                const unsigned done = atomicAdd(&S->field_done, 1u) + 1u;
                s_last = done == (unsigned)t.n_tiles_sys;
            }
        }
        __syncthreads();
        if (close_mode && s_last) {
            __threadfence();
            if (tid == T - 1) {
                // every tile of the system has folded its omega in: publish the
                // span (+inf when no bound is known) and reset the keys
                const uint32_t kx = atomicExch(&S->om_max_key, 0u);
                const uint32_t kn = atomicExch(&S->om_min_key, 0xFFFFFFFFu);
                const float span = kx >= kn ? __fsub_rn(ord_val(kx), ord_val(kn)) : INFINITY;
                S->omega_span = span >= 0.0f ? span : INFINITY;  // NaN (inf - inf): no bound
            }
            close_system(S, ef_part + t.first_tile, t.n_tiles_sys, mode, s_acc, s_ef);
            if (tid == 0) S->field_done = 0u;
        }
        __syncthreads();
    }
}

// Closes a launch for every system of the plan (one block per system): the
// sums of close_system over each system's tile ranges.
__global__ void __launch_bounds__(256) k_close(const SysClose* __restrict__ list, int n_sys,
                                                const double* __restrict__ ef_part, const double* __restrict__ eb_part,
                                                int mode) {
    __shared__ unsigned long long s_a[32];
    __shared__ double s_f[32];
    for (int si = blockIdx.x; si < n_sys; si += gridDim.x) {
        const SysClose L = list[si];
        if (mode & kCloseBond)
            close_system(L.sys, eb_part + L.move_first, L.move_count, mode, s_a, s_f);
        else
            close_system(L.sys, ef_part + L.field_first, L.field_count, mode, s_a, s_f);
    }
}

// The error words of the plan's systems in one word (one block).
__global__ void __launch_bounds__(256) k_error_words(const SysClose* __restrict__ list, int n_sys, uint32_t* out) {
    uint32_t any = 0u;
    for (int i = threadIdx.x; i < n_sys; i += blockDim.x) any |= list[i].sys->error_word;
    __shared__ uint32_t s_any[8];
    any = __reduce_or_sync(0xffffffffu, any);
    if ((threadIdx.x & 31) == 0) s_any[threadIdx.x >> 5] = any;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) any |= s_any[w];
        *out = any;
    }
}

// Bond energy sum_bonds k |r_i - r_j|^2 of the current positions, each bond
// once, one partial per tile (closed by k_close with kCloseBond).
__global__ void __launch_bounds__(256) k_bond_energy(const MoveTile* __restrict__ tiles, int n_tiles,
                                                      double* __restrict__ eb_part) {
    __shared__ double s_e[32];
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
    for (int ti = blockIdx.x; ti < n_tiles; ti += gridDim.x) {
        const MoveTile t = tiles[ti];
        SysDev* S = t.sys;
        const ArchDev* Ap = t.arch;
        const int L = Ap->length;
        const int nb = t.n_chains * L;
        const float* X = S->x + t.bead0;
        const float* Y = S->y + t.bead0;
        const float* Z = S->z + t.bead0;
        const float k = S->k;
        double e = 0.0;
        for (int i = tid; i < nb; i += T) {
            const int cl = (int)div_magic((uint32_t)i, Ap->len_magic, L);
            const int b = i - cl * L;
            const BeadInfo bi = Ap->beads[b];
            for (int d = 0; d < bi.deg; ++d) {
                const int j = bi.nbr[d];
                if (j <= b) continue;
                const int jj = cl * L + j;
                const float ex = X[i] - X[jj], ey = Y[i] - Y[jj], ez = Z[i] - Z[jj];
                e += (double)k * (double)(ex * ex + ey * ey + ez * ez);
            }
        }
        e = warp_sum(e);
        if (lane == 0) s_e[warp] = e;
        __syncthreads();
        if (tid == 0) {
            double a = 0.0;
            for (int w = 0; w < (T + 31) / 32; ++w) a += s_e[w];
            eb_part[ti] = a;
        }
        __syncthreads();
    }
}

// Adds the current counts into the time-averaged density accumulator and
// counts the sample (a sample taken outside the fused sweep).
__global__ void k_average_sample(SysDev* S, int64_t n) {
    const uint32_t* c32 = S->counts[S->cur];
    const uint16_t* c16 = reinterpret_cast<const uint16_t*>(c32);
    const bool half = S->count16 != 0;
    unsigned long long* avg = S->avg;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        avg[i] += half ? (unsigned long long)c16[i] : (unsigned long long)c32[i];
    if (blockIdx.x == 0 && threadIdx.x == 0) S->avg_samples += 1ull;
}

// Chain observables in double, one warp per chain and one partial row of
// kObsSlots sums per move tile (fixed reduction order).  Per chain:
// R_e = last bead - first bead (test.cpp:47-68 takes beads 0 and 31 of every
// chain); R_g^2 = mean |r - r_cm|^2; bonds counted once (j > i); with a
// reference snapshot, bead and centre-of-mass displacements.  Ana_Info
// (struct.h:65-75) names these analyses; the reference computes only R_e.
__global__ void __launch_bounds__(256) k_observables(const MoveTile* __restrict__ tiles, int n_tiles,
                                                      const float* __restrict__ ref, int64_t n_beads_sys,
                                                      double* __restrict__ part) {
    __shared__ double s_w[kMaxWarps][kObsSlots];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    for (int ti = blockIdx.x; ti < n_tiles; ti += gridDim.x) {
        const MoveTile t = tiles[ti];
        const SysDev* S = t.sys;
        const ArchDev* Ap = t.arch;
        const int L = Ap->length;
        double acc[kObsSlots];
#pragma unroll
        for (int k = 0; k < kObsSlots; ++k) acc[k] = 0.0;
        for (int cl = warp; cl < t.n_chains; cl += nwarps) {
            const int64_t b0 = t.bead0 + (int64_t)cl * L;
            const float* X = S->x + b0;
            const float* Y = S->y + b0;
            const float* Z = S->z + b0;
            double sx = 0.0, sy = 0.0, sz = 0.0, rx = 0.0, ry = 0.0, rz = 0.0;
            double bx = 0.0, by = 0.0, bz = 0.0, mx = 0.0, my = 0.0, mz = 0.0;
            for (int b = lane; b < L; b += 32) {
                const double x = X[b], y = Y[b], z = Z[b];
                sx += x; sy += y; sz += z;
                const BeadInfo bi = Ap->beads[b];
                for (int d = 0; d < bi.deg; ++d) {
                    const int j = bi.nbr[d];
                    if (j <= b) continue;
                    const double ex = (double)X[j] - x, ey = (double)Y[j] - y, ez = (double)Z[j] - z;
                    bx += ex * ex; by += ey * ey; bz += ez * ez;
                }
                if (ref) {
                    const double ux = x - (double)ref[b0 + b], uy = y - (double)ref[n_beads_sys + b0 + b],
                                 uz = z - (double)ref[2 * n_beads_sys + b0 + b];
                    mx += ux * ux; my += uy * uy; mz += uz * uz;
                    rx += (double)ref[b0 + b];
                    ry += (double)ref[n_beads_sys + b0 + b];
                    rz += (double)ref[2 * n_beads_sys + b0 + b];
                }
            }
            sx = warp_sum(sx); sy = warp_sum(sy); sz = warp_sum(sz);
            const double cx = sx / L, cy = sy / L, cz = sz / L;
            double gx = 0.0, gy = 0.0, gz = 0.0;
            for (int b = lane; b < L; b += 32) {
                const double ux = (double)X[b] - cx, uy = (double)Y[b] - cy, uz = (double)Z[b] - cz;
                gx += ux * ux; gy += uy * uy; gz += uz * uz;
            }
            gx = warp_sum(gx); gy = warp_sum(gy); gz = warp_sum(gz);
            bx = warp_sum(bx); by = warp_sum(by); bz = warp_sum(bz);
            if (ref) {
                mx = warp_sum(mx); my = warp_sum(my); mz = warp_sum(mz);
                rx = warp_sum(rx); ry = warp_sum(ry); rz = warp_sum(rz);
            }
            if (lane == 0) {
                const double ex = (double)X[L - 1] - (double)X[0], ey = (double)Y[L - 1] - (double)Y[0],
                             ez = (double)Z[L - 1] - (double)Z[0];
                acc[kObsRe] += ex * ex; acc[kObsRe + 1] += ey * ey; acc[kObsRe + 2] += ez * ez;
                acc[kObsRg] += gx / L; acc[kObsRg + 1] += gy / L; acc[kObsRg + 2] += gz / L;
                acc[kObsBond] += bx; acc[kObsBond + 1] += by; acc[kObsBond + 2] += bz;
                if (ref) {
                    acc[kObsMsd] += mx; acc[kObsMsd + 1] += my; acc[kObsMsd + 2] += mz;
                    const double dx = cx - rx / L, dy = cy - ry / L, dz = cz - rz / L;
                    acc[kObsMsdCom] += dx * dx; acc[kObsMsdCom + 1] += dy * dy; acc[kObsMsdCom + 2] += dz * dz;
                }
            }
        }
        if (lane == 0)
            for (int k = 0; k < kObsSlots; ++k) s_w[warp][k] = acc[k];
        __syncthreads();
        if (tid < kObsSlots) {
            double a = 0.0;
            for (int w = 0; w < nwarps; ++w) a += s_w[w][tid];
            part[(int64_t)ti * kObsSlots + tid] = a;
        }
        __syncthreads();
    }
}

// State checks of scmf_validate (counters in out[], no trap).
__global__ void k_validate_positions(const SysDev* S, int64_t n, unsigned long long* out) {
    unsigned long long bad = 0, far = 0;
    const float lim = 0x1p22f;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float x = S->x[i], y = S->y[i], z = S->z[i];
        if (!isfinite(x) || !isfinite(y) || !isfinite(z)) {
            ++bad;
            continue;
        }
        if (fabsf(x * S->inv_dx) >= lim || fabsf(y * S->inv_dy) >= lim || fabsf(z * S->inv_dz) >= lim) ++far;
    }
    bad = warp_sum(bad);
    far = warp_sum(far);
    if ((threadIdx.x & 31) == 0 && (bad | far)) {
        atomicAdd(out + 0, bad);
        atomicAdd(out + 1, far);
    }
}

__global__ void k_validate_cells(const SysDev* S, const uint32_t* a, const uint32_t* b, int64_t n_words,
                                 int64_t n_values, unsigned long long* out, unsigned long long* sums) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    unsigned long long diff = 0, bad = 0;
    for (int64_t i = i0; i < n_words; i += stride) diff += a[i] != b[i] ? 1ull : 0ull;
    for (int64_t i = i0; i < n_values; i += stride)
        if (!isfinite(S->omega[i])) ++bad;
    const bool c16 = S->count16 != 0;
    const uint16_t* a16 = reinterpret_cast<const uint16_t*>(a);
    const int64_t nc = S->n_cells;
    for (int t = 0; t < S->n_types; ++t) {
        unsigned long long v = 0;
        for (int64_t c = i0; c < nc; c += stride)
            v += c16 ? (unsigned long long)a16[t * nc + c] : (unsigned long long)a[t * nc + c];
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0 && v) atomicAdd(sums + t, v);
    }
    diff = warp_sum(diff);
    bad = warp_sum(bad);
    if ((threadIdx.x & 31) == 0 && (diff | bad)) {
        atomicAdd(out + 2, diff);
        atomicAdd(out + 3, bad);
    }
}

// ------------------------------------------------------------- transposes
__device__ __forceinline__ int64_t aos_bead_of(const SysDev* S, const ArchDev* archs, int n_arch, int64_t i) {
    int a = 0;
    while (a + 1 < n_arch && i >= archs[a + 1].bead_base) ++a;
    const ArchDev& A = archs[a];
    const int64_t r = i - A.bead_base;
    const int64_t slot_local = r / A.length;
    const int64_t b = r - slot_local * A.length;
    const uint32_t gc = S->chain_id[A.chain_base + slot_local];
    return A.bead_base + (int64_t)(gc - (uint32_t)A.rng_base) * A.length + b;
}

__global__ void k_aos_to_soa(const float* __restrict__ aos, SysDev* S, const ArchDev* archs, int n_arch,
                             int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t src = aos_bead_of(S, archs, n_arch, i);
        S->x[i] = aos[3 * src];
        S->y[i] = aos[3 * src + 1];
        S->z[i] = aos[3 * src + 2];
    }
}

__global__ void k_soa_to_aos(float* __restrict__ aos, const SysDev* S, const ArchDev* archs, int n_arch,
                             int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t dst = aos_bead_of(S, archs, n_arch, i);
        aos[3 * dst] = S->x[i];
        aos[3 * dst + 1] = S->y[i];
        aos[3 * dst + 2] = S->z[i];
    }
}

__global__ void k_unpack16(const SysDev* S, uint32_t* out, int64_t n) {
    const uint16_t* src = reinterpret_cast<const uint16_t*>(S->counts[S->cur]);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = src[i];
}

// ------------------------------------------------------------ diagnostics
__global__ void k_debug_math(uint32_t k0, uint32_t k1, int n, uint32_t* words, float* logs, float* normals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint4 w = philox4x32_10(make_uint4((uint32_t)i, 0u, 0u, 0u), k0, k1);
    words[4 * i] = w.x;
    words[4 * i + 1] = w.y;
    words[4 * i + 2] = w.z;
    words[4 * i + 3] = w.w;
    logs[i] = log_f(u01(w.w));
    float n0, n1, n2;
    normals3(w, normal_table(), n0, n1, n2);
    normals[3 * i] = n0;
    normals[3 * i + 1] = n1;
    normals[3 * i + 2] = n2;
}

// -------------------------------------------------------------- launchers
int launch_debug_math(uint32_t k0, uint32_t k1, int n, uint32_t* words, float* logs, float* normals, void* stream) {
    k_debug_math<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(k0, k1, n, words, logs, normals);
    return (int)cudaGetLastError();
}

int sm_count() {
    static std::mutex mu;
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    std::lock_guard<std::mutex> g(mu);
    if (cached[dev] == 0) {
        int n = 0;
        cached[dev] = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 148;
    }
    return cached[dev];
}

static int grid_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    const int64_t cap = (int64_t)sm_count() * 32;
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

// The statistics of the last sweep in the public layout (scmf_get_sweep_stats).
__global__ void k_stats_out(SysDev* S) {
    scmf_stats o;
    o.step = S->step;
    o.last_accepts = S->last_accepts;
    o.total_accepts = S->total_accepts;
    o.total_moves = S->total_moves;
    o.e_bond = S->e_bond_step == S->step + 1u ? S->e_bond : __longlong_as_double(0x7FF8000000000000ll);
    o.e_field = S->e_field;
    o.error_word = S->error_word;
    o.reserved = 0u;
    S->stats_out = o;
}

__global__ void k_copy_counts(const SysDev* __restrict__ S, uint32_t* __restrict__ dst, int64_t n) {
    const uint32_t* src = S->counts[S->cur];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

int launch_copy_counts(const SysDev* d_sys, uint32_t* dst, int64_t n_words, void* stream) {
    k_copy_counts<<<grid_for(n_words, 256), 256, 0, (cudaStream_t)stream>>>(d_sys, dst, n_words);
    return (int)cudaGetLastError();
}

int launch_stats_out(SysDev* d_sys, void* stream) {
    k_stats_out<<<1, 1, 0, (cudaStream_t)stream>>>(d_sys);
    return (int)cudaGetLastError();
}

int launch_init_coords(SysDev* d_sys, const ArchDev* d_arch, int n_arch, int n_chains, void* stream) {
    if (n_chains <= 0) return 0;
    const int th = 128;
    k_init_coords<<<(n_chains + th - 1) / th, th, 0, (cudaStream_t)stream>>>(d_sys, d_arch, n_arch, n_chains);
    return (int)cudaGetLastError();
}

template <bool ONE, int FORM, int KEYS>
static cudaError_t opt_in_form() {
    const auto opt_in = [](const void* f) {
        return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, SweepLayout<FORM>::kBytes);
    };
    const cudaError_t e = opt_in((const void*)k_sweep_warp<ONE, FORM, KEYS>);
    return e == cudaSuccess ? opt_in((const void*)k_run<ONE, FORM, KEYS>) : e;
}

template <bool ONE, int KEYS>
static cudaError_t opt_in_warp() {
    cudaError_t e = opt_in_form<ONE, kFormScreened, KEYS>();
    if (e == cudaSuccess) e = opt_in_form<ONE, kFormLong, KEYS>();
    if (e == cudaSuccess) e = opt_in_form<ONE, kFormUnscreened, KEYS>();
    if (e == cudaSuccess) e = opt_in_form<ONE, kFormGraph, KEYS>();
    return e;
}

template <bool ONE, int FOLD, int KEYS>
static cudaError_t opt_in_pairs() {
    return cudaFuncSetAttribute((const void*)k_sweep_pairs<ONE, FOLD, KEYS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                pairs_smem<ONE>());
}

int configure_kernels() {
    // once per device, with that device current
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaError_t e0 = cudaGetDevice(&dev);
    if (e0 != cudaSuccess) return (int)e0;
    std::lock_guard<std::mutex> g(mu);
    if (dev >= 0 && dev < 64 && done[dev]) return 0;
    int2 fold_tab[257] = {};
    for (int n = 2; n <= 256; ++n) fold_tab[n] = make_int2(fold_offset(n), (int)fold_magic_of(n));
    cudaError_t ef = cudaMemcpyToSymbol(c_fold, fold_tab, sizeof fold_tab);
    if (ef != cudaSuccess) return (int)ef;
    // opt the sweep kernels in to the largest dynamic shared memory, outside any stream capture
    const int bytes = (int)sweep_smem_bytes(kMaxTileBeads, kMaxLength);
    const auto opt_in = [](const void* f, int n) {
        return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, n);
    };
    const void* const general[] = {(const void*)k_sweep<kMoveOnly, kKeysNone>, (const void*)k_sweep<kMoveGrid, kKeysNone>,
                                   (const void*)k_sweep<kMoveOnly, kKeysHigh>, (const void*)k_sweep<kMoveGrid, kKeysHigh>,
                                   (const void*)k_sweep<kMoveOnly, kKeysBoth>, (const void*)k_sweep<kMoveGrid, kKeysBoth>};
    cudaError_t e = opt_in_warp<true, kKeysBoth>();
    if (e == cudaSuccess) e = opt_in_warp<false, kKeysHigh>();
    if (e == cudaSuccess) e = opt_in_warp<false, kKeysNone>();
    if (e == cudaSuccess) e = opt_in_pairs<true, 0, kKeysBoth>();
    if (e == cudaSuccess) e = opt_in_pairs<true, 1, kKeysBoth>();
    if (e == cudaSuccess) e = opt_in_pairs<true, 2, kKeysBoth>();
    if (e == cudaSuccess) e = opt_in_pairs<false, 3, kKeysHigh>();
    if (e == cudaSuccess) e = opt_in_pairs<false, 3, kKeysNone>();
    for (const void* f : general)
        if (e == cudaSuccess) e = opt_in(f, bytes);
    if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
    return (int)e;
}

template <int MODE>
static void launch_general(const MoveTile* tiles, int n_tiles, int blocks, int mtb, int ml, const LaunchShape& sh,
                           cudaStream_t st) {
    const size_t smem = sweep_smem_bytes(mtb, ml);
    if (sh.keyed == kKeysBoth)
        k_sweep<MODE, kKeysBoth><<<blocks, sh.threads, smem, st>>>(tiles, n_tiles, mtb, ml, sh.keys);
    else if (sh.keyed == kKeysHigh)
        k_sweep<MODE, kKeysHigh><<<blocks, sh.threads, smem, st>>>(tiles, n_tiles, mtb, ml, sh.keys);
    else
        k_sweep<MODE, kKeysNone><<<blocks, sh.threads, smem, st>>>(tiles, n_tiles, mtb, ml, sh.keys);
}

// A launch that may begin (set up its shared memory, wait) beside the last blocks of
// the kernel before, where `chained`.
template <typename... Args>
static cudaError_t launch_chained(void (*kernel)(Args...), int blocks, int threads, int smem, bool chained, cudaStream_t st,
                                  typename std::common_type<Args>::type... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// A launch over warp tiles in shared memory: k_sweep_warp, or k_run when `run` is given.
template <bool ONE, int FORM, int KEYS>
static cudaError_t launch_form(const SweepArgs& a, const RunArgs* run, bool chained, cudaStream_t st) {
    using Lay = SweepLayout<FORM>;
    const int sms = sm_count(), grid = a.n_tiles < sms ? a.n_tiles : sms;
    const int per_sm = (a.n_tiles + grid - 1) / grid, nw = per_sm < Lay::kWarps ? per_sm : Lay::kWarps;
    const int smem = Lay::kTabBytes + nw * (int)sizeof(typename Lay::Warp) + kSlack;
    if (!run) return launch_chained(k_sweep_warp<ONE, FORM, KEYS>, grid, 32 * nw, smem, chained, st, a);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;  // the blocks wait for one another
    at.val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(32u * (unsigned)nw);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_run<ONE, FORM, KEYS>, a, *run);
}

template <bool ONE, int KEYS>
static cudaError_t launch_warp(const SweepArgs& a, int form, const RunArgs* run, bool chained, cudaStream_t st) {
    if (form == kFormLong) return launch_form<ONE, kFormLong, KEYS>(a, run, chained, st);
    if (form == kFormUnscreened) return launch_form<ONE, kFormUnscreened, KEYS>(a, run, chained, st);
    if (form == kFormGraph) return launch_form<ONE, kFormGraph, KEYS>(a, run, chained, st);
    return launch_form<ONE, kFormScreened, KEYS>(a, run, chained, st);
}

template <bool ONE, int FOLD, int KEYS>
static cudaError_t launch_pairs(const SweepArgs& a, int warps, bool chained, cudaStream_t st) {
    const int sms = sm_count(), grid = a.n_tiles < sms ? a.n_tiles : sms;
    return launch_chained(k_sweep_pairs<ONE, FOLD, KEYS>, grid, 32 * warps, pairs_smem<ONE>(), chained, st, a);
}

static cudaError_t launch_warp(const LaunchShape& sh, bool move_counts, const RunArgs* run, cudaStream_t st) {
    SweepArgs a{};
    a.tiles = sh.warp_tiles;
    a.n_tiles = sh.n_warp_tiles;
    a.move_counts = move_counts;
    a.once = sh.once;
    a.keys = sh.keys;
    a.system = sh.system;
    a.sys = sh.sweep;
    a.n_arch = sh.n_arch;
    for (int i = 0; i < sh.n_arch; ++i) a.arch[i] = sh.arch[i];
    const int warps = kSweepForms[sh.form].warps;
    if (sh.form == kFormPairs) {
        if (a.sys.fold == 0) return launch_pairs<true, 0, kKeysBoth>(a, warps, sh.chained != 0, st);
        if (a.sys.fold == 1) return launch_pairs<true, 1, kKeysBoth>(a, warps, sh.chained != 0, st);
        return launch_pairs<true, 2, kKeysBoth>(a, warps, sh.chained != 0, st);
    }
    if (sh.form == kFormPairsList) {
        if (sh.keyed != kKeysNone) return launch_pairs<false, 3, kKeysHigh>(a, warps, sh.chained != 0, st);
        return launch_pairs<false, 3, kKeysNone>(a, warps, sh.chained != 0, st);
    }
    if (sh.one) return launch_warp<true, kKeysBoth>(a, sh.form, run, sh.chained != 0, st);
    if (sh.keyed != kKeysNone) return launch_warp<false, kKeysHigh>(a, sh.form, run, sh.chained != 0, st);
    return launch_warp<false, kKeysNone>(a, sh.form, run, sh.chained != 0, st);
}

int launch_run(const LaunchShape& sh, const RunArgs& run, void* stream) {
    return (int)launch_warp(sh, true, &run, (cudaStream_t)stream);
}

int launch_sweep(int mode, const MoveTile* tiles, int n_tiles, int mtb, int ml, const LaunchShape& sh, void* stream) {
    if (n_tiles <= 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    if (mtb > kMaxTileBeads || ml > kMaxLength || sh.threads > 256 || sh.threads < 32) return (int)cudaErrorInvalidValue;
    const int blocks = sh.blocks > 0 ? sh.blocks : n_tiles;
    if (mode == kGridOnly) {
        k_grid<<<blocks, sh.threads, 0, st>>>(tiles, n_tiles);
    } else if (sh.n_warp_tiles > 0) {
        return (int)launch_warp(sh, mode == kMoveGrid, nullptr, st);
    } else if (mode == kMoveOnly) {
        launch_general<kMoveOnly>(tiles, n_tiles, blocks, mtb, ml, sh, st);
    } else {
        launch_general<kMoveGrid>(tiles, n_tiles, blocks, mtb, ml, sh, st);
    }
    return (int)cudaGetLastError();
}

template <bool FUSED>
static void launch_field_t(int nt, const FieldTile* tiles, int n_tiles, int force_update, int blocks, int threads,
                           double* ef, int close_mode, bool chained, cudaStream_t st) {
    const auto k = nt == 2 ? k_field<FUSED, 2> : nt == 3 ? k_field<FUSED, 3> : nt == 1 ? k_field<FUSED, 1> : k_field<FUSED, 0>;
    launch_chained(k, blocks, threads, 0, chained, st, tiles, n_tiles, force_update, ef, close_mode);
}

int launch_field(bool fused, int force_update, const FieldTile* tiles, int n_tiles, LaunchShape sh, double* ef_part,
                 int close_mode, void* stream) {
    if (n_tiles <= 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    const int blocks = sh.blocks > 0 ? sh.blocks : n_tiles;
    const int threads = sh.threads > 256 ? 256 : sh.threads;
    if (fused)
        launch_field_t<true>(sh.n_types, tiles, n_tiles, force_update, blocks, threads, ef_part, close_mode, sh.chained != 0, st);
    else
        launch_field_t<false>(sh.n_types, tiles, n_tiles, force_update, blocks, threads, ef_part, close_mode, false, st);
    return (int)cudaGetLastError();
}

int launch_bond_energy(const MoveTile* tiles, int n_tiles, LaunchShape sh, double* eb_part, void* stream) {
    if (n_tiles <= 0) return 0;
    k_bond_energy<<<n_tiles, sh.threads > 256 ? 256 : sh.threads, 0, (cudaStream_t)stream>>>(tiles, n_tiles, eb_part);
    return (int)cudaGetLastError();
}

int launch_close(const SysClose* list, int n_sys, const double* ef_part, const double* eb_part, int mode, void* stream) {
    if (n_sys <= 0) return 0;
    k_close<<<n_sys < 1024 ? n_sys : 1024, 256, 0, (cudaStream_t)stream>>>(list, n_sys, ef_part, eb_part, mode);
    return (int)cudaGetLastError();
}

int launch_error_words(const SysClose* list, int n_sys, uint32_t* out, void* stream) {
    k_error_words<<<1, 256, 0, (cudaStream_t)stream>>>(list, n_sys, out);
    return (int)cudaGetLastError();
}

// One chunk of a chunked upload: positions of storage beads [i0, i1) (the
// AoS bead of storage bead i is bead i: chain ids are the identity plus each
// architecture's random-stream base) and their counts into counts[0].
__global__ void k_aos_chunk(const float* __restrict__ aos, SysDev* S, const ArchDev* archs, int n_arch, int64_t i0,
                            int64_t i1) {
    MoveConsts c;
    c.k = S->k; c.k2 = S->k2; c.A = S->A; c.R = S->R;
    c.inv_dx = S->inv_dx; c.inv_dy = S->inv_dy; c.inv_dz = S->inv_dz;
    load_fold(c, S);
    const int64_t NC = S->n_cells;
    uint32_t* cnt = S->counts[0];
    const bool c16 = S->count16 != 0;
    for (int64_t i = i0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < i1; i += (int64_t)gridDim.x * blockDim.x) {
        const float x = aos[3 * i], y = aos[3 * i + 1], z = aos[3 * i + 2];
        S->x[i] = x;
        S->y[i] = y;
        S->z[i] = z;
        int a = 0;
        while (a + 1 < n_arch && i >= archs[a + 1].bead_base) ++a;
        const ArchDev& A = archs[a];
        const int r = (int)(i - A.bead_base);  // systems hold fewer than 2^31 beads
        const int b = r % A.length;
        const int64_t idx = (int64_t)A.types[b] * NC + cell_of(c, x, y, z);
        if (c16)
            atomicAdd(cnt + (idx >> 1), 1u << ((idx & 1) * 16));
        else
            atomicAdd(cnt + idx, 1u);
    }
}

int launch_aos_chunk(const float* aos, SysDev* sys, const ArchDev* arch, int n_arch, int64_t i0, int64_t i1,
                     void* stream) {
    if (i1 <= i0) return 0;
    k_aos_chunk<<<grid_for(i1 - i0, 256), 256, 0, (cudaStream_t)stream>>>(aos, sys, arch, n_arch, i0, i1);
    return (int)cudaGetLastError();
}

int launch_aos_to_soa(const float* aos, SysDev* sys, const ArchDev* arch, int n_arch, int64_t n, void* stream) {
    if (n <= 0) return 0;
    k_aos_to_soa<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(aos, sys, arch, n_arch, n);
    return (int)cudaGetLastError();
}

int launch_soa_to_aos(float* aos, const SysDev* sys, const ArchDev* arch, int n_arch, int64_t n, void* stream) {
    if (n <= 0) return 0;
    k_soa_to_aos<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(aos, sys, arch, n_arch, n);
    return (int)cudaGetLastError();
}

int launch_unpack_counts16(const SysDev* sys, uint32_t* out, int64_t n, void* stream) {
    if (n <= 0) return 0;
    k_unpack16<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(sys, out, n);
    return (int)cudaGetLastError();
}
int launch_validate_positions(const SysDev* sys, int64_t n, unsigned long long* out, void* stream) {
    if (n <= 0) return 0;
    k_validate_positions<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(sys, n, out);
    return (int)cudaGetLastError();
}
int launch_validate_cells(const SysDev* sys, const uint32_t* a, const uint32_t* b, int64_t n_words, int64_t n_values,
                          unsigned long long* out, unsigned long long* sums, void* stream) {
    const int64_t n = n_words > n_values ? n_words : n_values;
    if (n <= 0) return 0;
    k_validate_cells<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(sys, a, b, n_words, n_values, out, sums);
    return (int)cudaGetLastError();
}
int launch_average_sample(SysDev* sys, int64_t n, void* stream) {
    if (n <= 0) return 0;
    k_average_sample<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(sys, n);
    return (int)cudaGetLastError();
}
int launch_observables(const MoveTile* tiles, int n_tiles, const float* ref_xyz, int64_t n_beads_sys, double* part,
                       void* stream) {
    if (n_tiles <= 0) return 0;
    k_observables<<<n_tiles, 256, 0, (cudaStream_t)stream>>>(tiles, n_tiles, ref_xyz, n_beads_sys, part);
    return (int)cudaGetLastError();
}

}  // namespace scmf

// ---------------------------------------------------------------------------
// Field update without allocation.
//
// For callers that cannot call cudaMalloc (code that runs where allocation is
// forbidden or must not stall, such as a step that is replayed inside someone
// else's captured stream work, or an embedding application that owns all
// device memory and hands out only pointers to its own buffers), the omega
// update of caller-owned counts into caller-owned omega is offered with its
// only scratch, the per-tile partial sums of the field energy, held in a fixed
// array in this library's device memory.  Every GPU that loads the library
// holds that array (kNoAllocMaxTiles doubles, 16 KiB) until the process exits.
namespace scmf {

constexpr int kNoAllocTileCells = 4096;  // cells of a tile at most
constexpr int kNoAllocMaxTiles = 2048;   // n_cells <= 2048 * 4096 = 8,388,608

static __device__ __align__(256) double g_noalloc_partials[kNoAllocMaxTiles];

struct FieldParams {
    int64_t n_cells;
    float scale;
    int n_types;
    int lit;
    float cf[kMaxTypes * kMaxTypes];
};

// One tile of cells per block: omega of every cell and the tile's field energy
// sum_T omega_T n_T into partials[tile] (no atomics).  Bound by memory: a
// counts word in and an omega out per cell and type.  NT > 0 (1 to 4 types,
// buffers on 16-byte boundaries, n_cells a multiple of 4): 16-byte loads and
// stores, the type count and the coefficients known as operands; NT = 0: any
// types and alignment, a cell at a time.  The tile is the smallest of 1,024, 2,048
// and 4,096 cells that the partials' array covers, so that 2.1M cells are 2,048
// blocks and every thread has its loads of all types in flight at once.  Two types
// on 2,097,152 cells (33.5 MB): 26.6 us with a cell at a time and tiles of 4,096,
// 6.6 us so, k_sum_partials included; 4,096 cells 12.7 and 3.0 us.
template <int NT>
__global__ void __launch_bounds__(256) k_field_noalloc(const uint32_t* __restrict__ counts, float* __restrict__ omega,
                                                        const __grid_constant__ FieldParams p, int tile_cells,
                                                        double* __restrict__ partials) {
    __shared__ double s_ef[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t c0 = (int64_t)blockIdx.x * tile_cells, c1 = min(c0 + (int64_t)tile_cells, p.n_cells);
    double ef = 0.0;
    float wmax = -INFINITY, wmin = INFINITY;  // not used: the caller's omega has no span slot
    if constexpr (NT > 0) {
        for (int64_t cell = c0 + 4 * tid; cell < c1; cell += 1024)
            ef += field_cells4<NT, false>(cell, p.n_cells, p.scale, p.lit != 0, true, counts, omega, p.cf, nullptr, wmax, wmin);
    } else {
        for (int64_t cell = c0 + tid; cell < c1; cell += 256)
            ef += field_cell<0, false>(p.n_types, cell, p.n_cells, p.scale, p.lit != 0, true, false, counts, omega, p.cf,
                                       nullptr, wmax, wmin);
    }
    ef = warp_sum(ef);
    if (lane == 0) s_ef[warp] = ef;
    __syncthreads();
    if (tid == 0) {
        double e = 0.0;
        for (int w = 0; w < 8; ++w) e += s_ef[w];
        partials[blockIdx.x] = e;
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // k_sum_partials may be set up
}

// Sum of the tile partials in a fixed order (one block).
// Launched as the field kernel's programmatic dependent: it waits here for that
// kernel's end, so only its own start overlaps.
__global__ void __launch_bounds__(256) k_sum_partials(const double* __restrict__ partials, int n,
                                                       double* __restrict__ out) {
    __shared__ double s_e[8];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    double e = 0.0;
    for (int i = threadIdx.x; i < n; i += 256) e += __ldcg(partials + i);
    e = warp_sum(e);
    if ((threadIdx.x & 31) == 0) s_e[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) e += s_e[w];
        *out = e;
    }
}

// The id of the calling thread's current CUDA context (0 when none is current
// or the driver cannot tell).  Taken through the driver entry points, so the
// library needs no link against libcuda.
static unsigned long long current_context_id() {
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, nullptr) == cudaSuccess)
            get_current = reinterpret_cast<GetCurrent>(f);
        f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, nullptr) == cudaSuccess)
            get_id = reinterpret_cast<GetId>(f);
    });
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// Device address of the scratch array for the current device.  The host-side
// name of a __device__ variable is only a stand-in for it and must never be
// passed to a kernel.  The address is looked up (with the device current) on
// the first call in a context and cached with that context's id; a context
// created later on the device (after cudaDeviceReset, or when the primary
// context was released and retained again) loads the module anew, so its id
// differs and the address is looked up again.  Without a context id from the
// driver it is looked up on every call.
static double* noalloc_scratch(int device, cudaError_t* err) {
    struct Entry {
        unsigned long long ctx;
        double* addr;
    };
    static std::mutex mu;
    static Entry cache[64] = {};
    if (device < 0 || device >= 64) {
        *err = cudaErrorInvalidDevice;
        return nullptr;
    }
    std::lock_guard<std::mutex> g(mu);
    const unsigned long long ctx = current_context_id();
    if (ctx != 0 && cache[device].ctx == ctx && cache[device].addr) {
        *err = cudaSuccess;
        return cache[device].addr;
    }
    void* p = nullptr;
    *err = cudaGetSymbolAddress(&p, g_noalloc_partials);
    if (*err != cudaSuccess) return nullptr;
    // the lookup makes the device's context current if none was: take its id now
    cache[device] = Entry{current_context_id(), static_cast<double*>(p)};
    return cache[device].addr;
}

}  // namespace scmf

// The entry point (declared in include/scmf.h).
extern "C" scmf_status scmf_update_omega_noalloc(const uint32_t* d_counts, float* d_omega, int32_t n_types,
                                                 int64_t n_cells, double field_scaling, const double* xn,
                                                 int32_t reference_nbeads, int32_t hamiltonian, double* d_energy,
                                                 void* stream) {
    using namespace scmf;
    if (!d_counts || !d_omega || !xn || !d_energy) return fail(SCMF_E_INVALID, "NULL argument");
    if (n_types < 1 || n_types > kMaxTypes) return fail(SCMF_E_INVALID, "n_types %d not in [1,%d]", n_types, kMaxTypes);
    if (n_cells < 1) return fail(SCMF_E_INVALID, "n_cells must be positive");
    if (n_cells > (int64_t)kNoAllocMaxTiles * kNoAllocTileCells)
        return fail(SCMF_E_INVALID,
                    "n_cells %lld exceeds the %lld cells the fixed scratch of the allocation-free field update covers",
                    (long long)n_cells, (long long)kNoAllocMaxTiles * kNoAllocTileCells);
    if (reference_nbeads < 1) return fail(SCMF_E_INVALID, "reference_nbeads must be >= 1");
    if (hamiltonian != SCMF_HAM_SCMF0 && hamiltonian != SCMF_HAM_LITERAL) return fail(SCMF_E_INVALID, "unknown hamiltonian");
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return fail(SCMF_E_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    double* scratch = noalloc_scratch(device, &e);
    if (!scratch) return fail(SCMF_E_CUDA, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
    FieldParams p{};
    p.n_cells = n_cells;
    p.scale = (float)field_scaling;
    p.n_types = n_types;
    p.lit = hamiltonian == SCMF_HAM_LITERAL;
    field_coefficients(n_types, xn, reference_nbeads, hamiltonian, p.cf);
    int tile = 1024;
    while (tile < kNoAllocTileCells && n_cells > (int64_t)kNoAllocMaxTiles * tile) tile *= 2;
    const int tiles = (int)((n_cells + tile - 1) / tile);
    const bool vec = n_types <= 4 && n_cells % 4 == 0 && (((uintptr_t)d_counts | (uintptr_t)d_omega) & 15) == 0;
    cudaStream_t st = (cudaStream_t)stream;
    const auto k = !vec           ? k_field_noalloc<0>
                   : n_types == 1 ? k_field_noalloc<1>
                   : n_types == 2 ? k_field_noalloc<2>
                   : n_types == 3 ? k_field_noalloc<3>
                                  : k_field_noalloc<4>;
    k<<<tiles, 256, 0, st>>>(d_counts, d_omega, p, tile, scratch);
    e = cudaGetLastError();
    if (e == cudaSuccess) {
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(1);
        cfg.blockDim = dim3(256);
        cfg.stream = st;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, k_sum_partials, (const double*)scratch, tiles, d_energy);
    }
    if (e != cudaSuccess) return fail(SCMF_E_CUDA, "launch: %s", cudaGetErrorString(e));
    return SCMF_OK;
}
