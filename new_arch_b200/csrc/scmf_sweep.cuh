// The move on warp tiles: k_sweep_warp (one sweep's move of any systems),
// k_sweep_pairs (of systems that are not screened) and k_run (many whole sweeps of
// systems that fit on the chip); included by scmf_kernels.cu.
//
// What a sweep costs is arithmetic: every trial needs its Philox block (twenty
// 32 x 32 -> 64 bit products, four cycles of a scheduler's multiplier each),
// three normals, a force and an energy, about 200 warp instructions in all, while
// its bytes take a third of that time.  Where proposals overshoot (A 4k of
// several, the synthetic workloads: one trial in two hundred accepted) nearly all
// of this proves a rejection that a coarser computation can prove too.  So a
// sweep is split:
//
//  * screen: every trial is proposed with its own Philox block but with normals
//    from a small piecewise-linear table, and rejected when the energy that
//    even the table's error leaves cannot pass the Metropolis test whatever
//    omega holds (ScreenDev has the inequality).  The even and the odd bead of a
//    pair run side by side, as the halves of packed f32x2 operations, and share
//    the first Philox rounds.  The loop takes 141 cycles of a scheduler per
//    warp of trials, half of them Philox's, from four warps a scheduler on
//    (16, 24, 28 and 32 warps an SM measure the same).
//  * resolve: the trials left over (2.8 % in the large system) are gathered into
//    a list of the warp and made exactly, a full warp at a time: exact normals,
//    energy, cells, omega, Metropolis, with the words of the general kernel.
//    Even beads first; every odd neighbour of an even bead that moved, whose
//    screen saw the old position, is added to the odd beads' list.
//
// A system whose proposals mostly pass (ScreenLevel: the reference's own units)
// skips the screen and resolves every trial, here or in k_sweep_pairs.  Either way positions and
// counts are the ones that the oracle gives, bit for bit.
//
// Each warp has tiles of its own (up to SweepLayout::kBeads beads in its part of shared
// memory) and waits for no other warp.  Measured against this on the large system
// (51.2M beads, 0.326 ms): warps that only screen beside warps that only resolve
// 0.375 ms (an exact trial waits for positions, table and omega, but mostly it
// takes its share of the same pipes); the trials of several tiles resolved
// together from global memory 0.344 ms; 20 warps with smaller tiles 0.324 ms.
// The kernels before it (a thread per bead pair in registers, every trial exact)
// took 0.379 ms, and 0.051 ms for 2.0M beads in chains of 33 where this takes
// 0.025 ms.
#pragma once
#include <stddef.h>

#include <type_traits>

#include "scmf_screen_table.h"

namespace scmf {

// ---------------------------------------------------------- packed fp32 pairs
// Two rounded-to-nearest FP32 operations in one instruction (sm_100).  The
// same bits as the scalar operations on each half.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// ------------------------------------------------------ bulk copies, barriers
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0u;
}
// Waits for a phase of a barrier of this CTA; false after kWaitClocks (never in a sound
// run).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    do {
        if (mbar_try(bar, parity)) return true;
    } while (clock64() - t0 < kWaitClocks);
    return false;
}
// A bulk copy from global memory whose lines leave L2 before others where
// `once` is set: positions that are read once a sweep, when they are more than L2
// holds, would push omega and the counts out.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, bool once) {
    uint64_t policy;
    if (once)
        asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    else
        asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(policy));
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar), "l"(policy)
        : "memory");
}
// Orders this thread's earlier accesses before later bulk copies.
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

// ------------------------------------------------------------------- layout
constexpr int kScreenCopies = 16;
constexpr int kListLen = 128;
constexpr int kSlack = 256;  // the lanes past a tile's last pair read up to 64 words past its buffer
constexpr int kTilePad = 12;  // 4 words before the tile, its offset of up to 3, and 2 read past its last pair
// The screen table follows the exact normal table: kScreenCopies lane-
// interleaved copies (lane l reads copy l mod 16: the half warps of an 8-byte
// read then meet no bank twice).
constexpr int kScreenTabAt = SCMF_NORMAL_SEGS * (int)sizeof(float4);
constexpr int sweep_tab_bytes(int form) {
    return kScreenTabAt + (form == kFormUnscreened ? 0 : SCMF_SCREEN_SEGS * kScreenCopies * (int)sizeof(float2));
}

// A CTA's warps and what each has in shared memory, for each SweepFormId.
template <int FORM>
struct SweepLayout {
    static constexpr int kWarps = kSweepForms[FORM].warps;
    static constexpr int kBeads = kSweepForms[FORM].beads;
    static constexpr int kStride = kBeads + kTilePad;  // from x to y to z
    struct Warp {
        uint64_t full;         // barrier: the tile has arrived
        uint64_t pad;
        uint32_t moved[32];    // odd beads next to an even bead that moved: a bit for each row, a word for each lane
        uint16_t list[kListLen];
        SweepSys sys;          // of the tile's system, where a launch has several
        BondConsts by_deg[FORM == kFormGraph ? kGraphDeg + 1 : 1];  // SysDev's
        // k_run, which has registers for one phase of a sweep at a time: the warp's
        // tile and its architecture, the sweeps that its system has made and makes
        // in all, and the warp's field tile and its system
        struct {
            WarpTile tile;
            const uint8_t* types;
            uint32_t rng_base, h_magic, base, stop;
            int32_t rule, active;
            SysDev* f_sys;
            int64_t cell0;
            int32_t n_cells;
            uint32_t f_base, f_stop;
        } run;
        FieldSys field;
        alignas(16) float pos[3 * kStride];
    };
    static constexpr int kTabBytes = sweep_tab_bytes(FORM);
    static constexpr int kBytes = kTabBytes + kWarps * (int)sizeof(Warp) + kSlack;
    static_assert(kTilePairs <= 32 * 32, "a row of 32 bead pairs is a bit of a lane's mask");
    static_assert(kTabBytes % 16 == 0 && sizeof(Warp) % 16 == 0 && offsetof(Warp, pos) % 16 == 0 && kStride % 4 == 0,
                  "16-byte copies");
    static_assert(kBytes <= 227 * 1024, "shared memory of an SM");
};

// ------------------------------------------------------------------- screen
// A normal of word w to within SCMF_SCREEN_DELTA, times 2^30.  lane_at is the
// byte offset of the lane's copy in an entry (bits 3 to 6).
__device__ __forceinline__ float screen_normal(uint32_t w, uint32_t lane_at) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const float f = __uint2float_rn(w + w + 1u);
    const uint32_t at = ((__float_as_uint(f) >> 14) & 0xFFFFFF80u) | lane_at;  // (bits >> 21) * 16 copies * 8 bytes
    const float2 c = *reinterpret_cast<const float2*>(smem_raw + (kScreenTabAt - (127 << 2) * kScreenCopies * 8) + at);
    const float z = __fmaf_rn(c.y, f, c.x);
    return __uint_as_float(__float_as_uint(z) ^ (w & 0x80000000u));
}
__device__ __forceinline__ uint32_t screen_lane() { return (uint32_t)(threadIdx.x & (kScreenCopies - 1)) * 8u; }

// log2 of a value that lies below the uniform of word w (u01 drops the low
// nine bits of w; the conversion and the subtraction round by at most 2^-25
// each): -inf or NaN for the smallest uniforms, which then pass the screen.
__device__ __forceinline__ float log2_below_u(uint32_t w) {
    const float u = __fmaf_rn(__uint2float_rn(w), -0x1p-32f, 0x1.fffffcp-1f);
    float l;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(u));
    return l;
}

// The Philox blocks of the two beads of a pair, with the work that they share
// (the chain and step words) done once: (chain, b, step, 0) and (chain, b + 1,
// step, 0).  PairHead is what depends on the beads and the step alone.
struct PairHead {
    uint32_t y1;                  // low word of M1 * step
    uint64_t p0e, p0o;            // M0 * x of round 1, for the even and the odd bead
};
template <int KEYS>
__device__ __forceinline__ PairHead pair_head(uint32_t b, uint32_t step, uint32_t k0, const PhiloxKeys& ks) {
    const uint64_t m1s = (uint64_t)0xCD9E8D57u * step;
    const uint32_t hi = (uint32_t)(m1s >> 32) ^ (KEYS == kKeysBoth ? ks.k[0] : k0);
    PairHead h;
    h.y1 = (uint32_t)m1s;
    h.p0e = (uint64_t)0xD2511F53u * (hi ^ b);
    h.p0o = (uint64_t)0xD2511F53u * (hi ^ (b + 1u));
    return h;
}
template <int KEYS>
__device__ __forceinline__ void pair_blocks(uint32_t chain, const PairHead& h, uint32_t k0, uint32_t k1,
                                            const PhiloxKeys& ks, uint4& we, uint4& wo) {
    // the key words of round r (KeyMode: from the schedule, or advanced here)
    const auto key0 = [&](int r) { return KEYS == kKeysBoth ? ks.k[2 * r] : k0; };
    const auto key1 = [&](int r) { return KEYS != kKeysNone ? ks.k[2 * r + 1] : k1; };
    const auto next = [&] {
        if (KEYS != kKeysBoth) k0 += 0x9E3779B9u;
        if (KEYS == kKeysNone) k1 += 0xBB67AE85u;
    };
    const uint64_t a = (uint64_t)0xD2511F53u * chain;                                   // round 1
    const uint64_t q = (uint64_t)0xCD9E8D57u * ((uint32_t)(a >> 32) ^ key1(0));         // round 2
    next();
    const uint32_t x2 = (uint32_t)(q >> 32) ^ h.y1 ^ key0(1);
    we.z = (uint32_t)(h.p0e >> 32) ^ (uint32_t)a ^ key1(1);
    wo.z = (uint32_t)(h.p0o >> 32) ^ (uint32_t)a ^ key1(1);
    next();
    const uint64_t c = (uint64_t)0xD2511F53u * x2;                                      // round 3
    const uint64_t de = (uint64_t)0xCD9E8D57u * we.z, d_o = (uint64_t)0xCD9E8D57u * wo.z;
    we = make_uint4((uint32_t)(de >> 32) ^ (uint32_t)q ^ key0(2), (uint32_t)de,
                    (uint32_t)(c >> 32) ^ (uint32_t)h.p0e ^ key1(2), (uint32_t)c);
    wo = make_uint4((uint32_t)(d_o >> 32) ^ (uint32_t)q ^ key0(2), (uint32_t)d_o,
                    (uint32_t)(c >> 32) ^ (uint32_t)h.p0o ^ key1(2), (uint32_t)c);
#pragma unroll
    for (int r = 3; r < 10; ++r) {
        next();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            uint4& w = i ? wo : we;
            const uint64_t p0 = (uint64_t)0xD2511F53u * w.x, p1 = (uint64_t)0xCD9E8D57u * w.z;
            w = make_uint4((uint32_t)(p1 >> 32) ^ w.y ^ key0(r), (uint32_t)p1,
                           (uint32_t)(p0 >> 32) ^ w.w ^ key1(r), (uint32_t)p0);
        }
    }
}

// Constants of a pair's two trials (even bead, odd bead).
struct PairConsts {
    f32x2 k2l, k2r;  // spring constants of the left and right bond, 0 where there is none; the odd bead's left
                     // one is negated (its difference is the even bead's right one)
    f32x2 a, b;      // ScreenDev's a and b
    // keeps the values in registers through the loop that follows
    __device__ __forceinline__ void pin() { asm volatile("" : "+l"(k2l), "+l"(k2r), "+l"(a), "+l"(b)); }
};
// What a warp keeps of the system and architecture that it is at.
struct SweepConsts {
    int L, h;                       // beads and pairs (ceil(L / 2)) of a chain
    uint32_t h_magic;               // div_magic of h
    uint32_t step, k0, k1;          // the sweep being made, the seed
    float k2, a1, a2, b1, b2, add;  // ScreenDev's, for beads of one and two bonds
    float u0, u1;                   // (4 / A)(span + 2^-18) and -(4 / A) ln 2: span + L of ScreenDev times 4 / A
    PairConsts pc;                  // KIND 0: the lane's
    PairHead head;
};
// first: the even bead starts its chain; single: it also ends it (no odd bead); last: the odd bead ends it.
__device__ __forceinline__ PairConsts pair_consts(const SweepConsts& s, bool first, bool single, bool last) {
    const bool e1 = first || single;
    PairConsts c;
    c.k2l = pack2(first ? 0.0f : s.k2, -s.k2);
    c.k2r = pack2(single ? 0.0f : s.k2, last ? 0.0f : s.k2);
    c.a = pack2(e1 ? s.a1 : s.a2, last ? s.a1 : s.a2);
    c.b = pack2(e1 ? s.b1 : s.b2, last ? s.b1 : s.b2);
    return c;
}

// The lane's pairs of a tile of `items` pairs (kTilePairs at most): bit i for pair 32 i + lane.
__device__ __forceinline__ uint32_t row_mask(int items) {
    const int n = max(0, (items - (int)(threadIdx.x & 31) + 31) >> 5);
    return n >= 32 ? 0xFFFFFFFFu : (1u << n) - 1u;
}

// Screens a tile: bit i of even (odd): the trial of the even (odd) bead of pair
// 32 i + lane may be accepted.  X is the first bead's x.
//   KIND 0: even L, h divides 32 (a lane's place in its chain never changes); 1:
//   even L; 2: odd L, or a tile whose first bead is at an odd offset.
template <int KIND, int FORM, int KEYS>
__device__ __forceinline__ void screen_tile(const SweepConsts& s, const float* X, uint32_t rng0, int n_chains,
                                            const PhiloxKeys& keys, uint32_t tab, uint32_t& even_out, uint32_t& odd_out) {
    using Lay = SweepLayout<FORM>;
    const int lane = threadIdx.x & 31;
    const int L = s.L, h = s.h, items = n_chains * h;
    uint32_t bit = 1u, even = 0u, odd = 0u;
    const uint32_t step = s.step, k0 = s.k0, k1 = s.k1, h_magic = s.h_magic;
    const float u0 = s.u0, u1 = s.u1;
    const f32x2 add = pack2(s.add, s.add);
    PairConsts pc = s.pc;
    PairHead head = s.head;
    if (KIND == 0) pc.pin();
    const float* P0 = X + 2 * lane;  // KIND 0: the lane's chain and place advance by constants
    uint32_t gc0 = KIND == 0 ? rng0 + div_magic((uint32_t)lane, h_magic, h) : 0u;
    const uint32_t gc_step = KIND == 0 ? 32u / (uint32_t)h : 0u;
#pragma unroll 1
    for (int j0 = 0; j0 < items; j0 += 32, bit += bit, P0 += 64, gc0 += gc_step) {
        int j = j0 + lane;
        if (KIND == 2) j = min(j, items - 1);
        const int cl = KIND == 0 ? 0 : (int)div_magic((uint32_t)j, h_magic, h);
        const int k = KIND == 0 ? 0 : j - cl * h;
        const float* const PX = KIND == 2 ? X + (cl * L + 2 * k) : P0;
        const uint32_t gc = KIND == 0 ? gc0 : rng0 + (uint32_t)cl;
        const bool single = KIND == 2 && 2 * k + 1 >= L;  // the pair has no odd bead
        if (KIND != 0) {
            pc = pair_consts(s, k == 0, single, KIND == 2 ? 2 * k + 2 >= L : k == h - 1);
            head = pair_head<KEYS>(2u * (uint32_t)k, step, k0, keys);
        }
        f32x2 f[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float* P = PX + a * Lay::kStride;
            float e, o;
            if (KIND == 2) {
                e = P[0];
                o = P[1];
            } else {
                const float2 v = *reinterpret_cast<const float2*>(P);
                e = v.x;
                o = v.y;
            }
            // the forces of the trial kernels, left bond then right bond; the
            // odd bead's left difference is the even bead's right one negated
            const float d = __fsub_rn(o, e), dl = __fsub_rn(P[-1], e), dr = __fsub_rn(P[2], o);
            f[a] = fma2(pack2(d, dr), pc.k2r, mul2(pack2(dl, d), pc.k2l));
        }
        uint4 we, wo;
        pair_blocks<KEYS>(gc, head, k0, k1, keys, we, wo);
        const f32x2 vx = fma2(f[0], pc.a, pack2(screen_normal(we.x, tab), screen_normal(wo.x, tab)));
        const f32x2 vy = fma2(f[1], pc.a, pack2(screen_normal(we.y, tab), screen_normal(wo.y, tab)));
        const f32x2 vz = fma2(f[2], pc.a, pack2(screen_normal(we.z, tab), screen_normal(wo.z, tab)));
        const f32x2 q = fma2(vx, vx, fma2(vy, vy, mul2(vz, vz)));
        const f32x2 u = pack2(__fmaf_rn(log2_below_u(accept_word(we)), u1, u0), __fmaf_rn(log2_below_u(accept_word(wo)), u1, u0));
        const f32x2 lim = fma2(pc.b, fma2(f[0], f[0], fma2(f[1], f[1], fma2(f[2], f[2], u))), add);
        float qe, qo, le, lo;
        unpack2(q, qe, qo);
        unpack2(lim, le, lo);
        if (!(qe > le)) even += bit;  // NaN passes
        if (!(qo > lo) && !single) odd += bit;
    }
    const uint32_t valid = row_mask(items);
    even_out = even & valid;
    odd_out = odd & valid;
}

// The cell of a position.
__device__ __forceinline__ int cell_index(const SweepSys& c, float x, float y, float z) {
    int ix, iy, iz;
    if (c.fold == 0) {
        ix = fold_pow2(x, c.inv_d[0], c.n[0] - 1);
        iy = fold_pow2(y, c.inv_d[1], c.n[1] - 1);
        iz = fold_pow2(z, c.inv_d[2], c.n[2] - 1);
    } else if (c.fold == 1) {
        ix = fold_magic(x, c.inv_d[0], c.n[0], c.fold_off[0], c.fold_mag[0]);
        iy = fold_magic(y, c.inv_d[1], c.n[1], c.fold_off[1], c.fold_mag[1]);
        iz = fold_magic(z, c.inv_d[2], c.n[2], c.fold_off[2], c.fold_mag[2]);
    } else {
        ix = fold(x, c.inv_d[0], c.n[0]);
        iy = fold(y, c.inv_d[1], c.n[1]);
        iz = fold(z, c.inv_d[2], c.n[2]);
    }
    return ix + c.n[0] * (iy + c.n[1] * iz);
}

// What the exact trials of a tile need besides the system.
struct TileRef {
    float* X;                // the first bead's x in the buffer
    int64_t bead0;           // its index in the system
    uint32_t rng0;           // random-stream id of the first chain
    int items;               // bead pairs
    const uint8_t* types;
    float span;
    bool move_counts;
    bool write;              // moved beads go to global memory too (k_run: after the last sweep)
};

// What a trial is made of: its random stream, the bead (its place p in the
// tile, its type's omega), the force on it, and c and A c / 4 of its bonds.
struct Trial {
    uint32_t chain, bead, typ;
    int p;
    float x, y, z, fx, fy, fz, cc, ac4;
};

// Makes a lane's trial exactly (where act), with trial_f's expressions.  A move
// updates the tile and, where asked, the positions in global memory, and moves a
// count if it leaves its cell.  Returns whether the bead moved.
template <int FORM, int KEYS>
__device__ __forceinline__ bool settle(const SweepSys& c, const SweepConsts& s, const TileRef& t, const PhiloxKeys& keys,
                                       const float4* ntab, const Trial& b, bool act) {
    constexpr int kStride = SweepLayout<FORM>::kStride;
    const uint4 w = philox_block<KEYS>(make_uint4(b.chain, b.bead, s.step, 0u), s.k0, s.k1, keys);
    float n0, n1, n2;
    normals3(w, ntab, n0, n1, n2);
    const float dx = __fmaf_rn(c.A, b.fx, __fmul_rn(c.R, n0));
    const float dy = __fmaf_rn(c.A, b.fy, __fmul_rn(c.R, n1));
    const float dz = __fmaf_rn(c.A, b.fz, __fmul_rn(c.R, n2));
    const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
    const float fd = __fmaf_rn(b.fx, dx, __fmaf_rn(b.fy, dy, __fmul_rn(b.fz, dz)));
    const float deb = __fmul_rn(b.ac4, __fmaf_rn(b.cc, d2, __fmul_rn(-2.0f, fd)));
    const float u = u01(accept_word(w));
    const float lo = log_lower(u);
    if (!(act && maybe_accepted(deb, t.span, lo))) return false;
    const float px = __fadd_rn(b.x, dx), py = __fadd_rn(b.y, dy), pz = __fadd_rn(b.z, dz);
    const int c_old = cell_index(c, b.x, b.y, b.z), c_new = cell_index(c, px, py, pz);
    const float w_old = __ldcg(c.omega + (b.typ + c_old)), w_new = __ldcg(c.omega + (b.typ + c_new));
    const float dE = __fadd_rn(__fsub_rn(w_new, w_old), deb);
    // log_lower decides without the logarithm for all but a few trials (trial_f)
    if (!(dE < 0.0f || (-dE > lo && log_f(u) < -dE))) return false;
    float* const Q = t.X + b.p;
    Q[0] = px;
    Q[kStride] = py;
    Q[2 * kStride] = pz;
    if (t.write) {
        const int64_t g = t.bead0 + b.p;
        c.x[g] = px;
        c.y[g] = py;
        c.z[g] = pz;
    }
    if (t.move_counts && c_new != c_old) count_move(c.counts, c.count16 != 0, b.typ, c_old, c_new);
    return true;
}

// The exact trial of the bead of parity par of a lane's pair (where act).  A bead
// that moves marks the odd beads next to it, whose screen saw the old position.
template <int FORM, int KEYS>
__device__ __forceinline__ unsigned exact_trial(const SweepSys& c, const SweepConsts& s, const TileRef& t, uint32_t* moved,
                                                const PhiloxKeys& keys, const float4* ntab, int par, int pair, bool act) {
    constexpr int kStride = SweepLayout<FORM>::kStride;
    const int cl = (int)div_magic((uint32_t)pair, s.h_magic, s.h);
    int bead = 2 * (pair - cl * s.h) + par;
    act = act && bead < s.L;
    bead = act ? bead : 0;
    Trial b;
    b.chain = t.rng0 + (uint32_t)cl;
    b.bead = (uint32_t)bead;
    b.p = cl * s.L + bead;
    b.typ = (uint32_t)__ldg(t.types + bead) * c.n_cells;
    const bool has_l = bead > 0, has_r = bead + 1 < s.L;
    const int l = has_l ? -1 : 0, r = has_r ? 1 : 0;  // a missing bond: the bead itself, and no spring
    const float* const Q = t.X + b.p;
    b.x = Q[0];
    b.y = Q[kStride];
    b.z = Q[2 * kStride];
    const float kl = has_l ? c.k2 : 0.0f, kr = has_r ? c.k2 : 0.0f;
    b.fx = b.fy = b.fz = 0.0f;
    add_bond(kl, b.x, b.y, b.z, Q[l], Q[l + kStride], Q[l + 2 * kStride], b.fx, b.fy, b.fz);
    add_bond(kr, b.x, b.y, b.z, Q[r], Q[r + kStride], Q[r + 2 * kStride], b.fx, b.fy, b.fz);
    const int deg = (has_l ? 1 : 0) + (has_r ? 1 : 0);
    b.cc = deg == 2 ? c.cdeg[2] : deg == 1 ? c.cdeg[1] : 0.0f;
    b.ac4 = deg == 2 ? c.ac4[2] : deg == 1 ? c.ac4[1] : 0.0f;
    if (!settle<FORM, KEYS>(c, s, t, keys, ntab, b, act)) return 0u;
    if (FORM != kFormUnscreened && par == 0) {
        if (bead > 0) atomicOr(moved + ((pair - 1) & 31), 1u << ((pair - 1) >> 5));
        if (bead + 1 < s.L) atomicOr(moved + (pair & 31), 1u << (pair >> 5));
    }
    return 1u;
}

// Makes the trials of a tile that the masks name (bit i of even / odd: the even
// / odd bead of pair 32 i + lane).  Returns the lane's accepted moves.
template <int FORM, int KEYS>
__device__ __forceinline__ unsigned resolve_tile(typename SweepLayout<FORM>::Warp* wp, const SweepSys& c, const SweepConsts& s,
                                                 const TileRef& t, const PhiloxKeys& keys, const float4* ntab, uint32_t even,
                                                 uint32_t odd) {
    const int lane = threadIdx.x & 31;
    unsigned nacc = 0;
    uint32_t mask = even;
#pragma unroll 1
    for (int par = 0; par < 2; ++par) {
        if (FORM == kFormUnscreened) {
            mask = par ? odd : even;
        } else if (par) {  // the odd neighbours of the even beads that moved
            mask = odd | wp->moved[lane];
            wp->moved[lane] = 0u;
        }
        if (FORM == kFormUnscreened) {  // every trial, row by row
#pragma unroll 1
            for (int r = 0; 32 * r < t.items; ++r) {
                nacc += exact_trial<FORM, KEYS>(c, s, t, wp->moved, keys, ntab, par, min(32 * r + lane, t.items - 1),
                                                ((mask >> r) & 1u) != 0u);
            }
            __syncwarp();
            continue;
        }
        const int own = __popc(mask);
        int before = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += v;
        }
        const int total = __shfl_sync(0xffffffffu, before, 31);
        if (2 * total <= t.items && total <= kListLen) {  // the pairs, gathered into full warps
            uint16_t* at = wp->list + (before - own);
            for (uint32_t m = mask; m; m &= m - 1u) *at++ = (uint16_t)((__ffs(m) - 1) * 32 + lane);
            __syncwarp();
#pragma unroll 1
            for (int r = lane; r < total; r += 32) {
                nacc += exact_trial<FORM, KEYS>(c, s, t, wp->moved, keys, ntab, par, (int)wp->list[r], true);
            }
        } else {  // row by row
#pragma unroll 1
            for (int r = 0; 32 * r < t.items; ++r) {
                nacc += exact_trial<FORM, KEYS>(c, s, t, wp->moved, keys, ntab, par, min(32 * r + lane, t.items - 1),
                                                ((mask >> r) & 1u) != 0u);
            }
        }
        __syncwarp();
    }
    return nacc;
}

// --------------------------------------------------------- other bond graphs
// A bead's GraphBead.
struct GraphRec {
    uint4 v;
    __device__ __forceinline__ uint32_t bead() const { return v.x & 0xFFFFu; }
    __device__ __forceinline__ int deg() const { return (int)((v.x >> 16) & 0xFFu); }
    __device__ __forceinline__ uint32_t type() const { return v.x >> 24; }
    __device__ __forceinline__ int nbr(int d) const {
        const uint32_t w = d < 2 ? v.y : d < 4 ? v.z : v.w;
        return (int)(d & 1 ? w >> 16 : w & 0xFFFFu);
    }
};
__device__ __forceinline__ GraphRec graph_rec(const GraphBead* beads, int k) {
    return GraphRec{__ldg(reinterpret_cast<const uint4*>(beads) + k)};
}

// The Philox block of bead b of a chain: pair_blocks for one bead (p0 = M0 * x of
// round 1, which the bead and the step give).
template <int KEYS>
__device__ __forceinline__ uint4 bead_block(uint32_t chain, uint32_t y1, uint64_t p0, uint32_t k0, uint32_t k1,
                                            const PhiloxKeys& ks) {
    const auto key0 = [&](int r) { return KEYS == kKeysBoth ? ks.k[2 * r] : k0; };
    const auto key1 = [&](int r) { return KEYS != kKeysNone ? ks.k[2 * r + 1] : k1; };
    const auto next = [&] {
        if (KEYS != kKeysBoth) k0 += 0x9E3779B9u;
        if (KEYS == kKeysNone) k1 += 0xBB67AE85u;
    };
    const uint64_t a = (uint64_t)0xD2511F53u * chain;                            // round 1
    const uint64_t q = (uint64_t)0xCD9E8D57u * ((uint32_t)(a >> 32) ^ key1(0));  // round 2
    next();
    uint4 w = make_uint4((uint32_t)(q >> 32) ^ y1 ^ key0(1), (uint32_t)q, (uint32_t)(p0 >> 32) ^ (uint32_t)a ^ key1(1),
                         (uint32_t)p0);
#pragma unroll
    for (int r = 2; r < 10; ++r) {
        next();
        const uint64_t m0 = (uint64_t)0xD2511F53u * w.x, m1 = (uint64_t)0xCD9E8D57u * w.z;
        w = make_uint4((uint32_t)(m1 >> 32) ^ w.y ^ key0(r), (uint32_t)m1, (uint32_t)(m0 >> 32) ^ w.w ^ key1(r), (uint32_t)m0);
    }
    return w;
}

// One sweep of a tile of chains of any bond graph, colour by colour: beads of one
// colour have no bond with each other, so a colour's trials are screened, gathered
// and made exactly before the next colour's are looked at, and no screen sees a
// position that moves.  Without the screen every trial is made.  Returns the
// lane's accepted moves.
//
// The screen takes 64 trials a step, two a lane, as the halves of f32x2
// operations.  A lane keeps its two beads from step to step while the chains
// advance (ArchDev::color_width beads of color_per chains a step: at least half of
// the lanes, and 60 of 64 for twenty beads of a colour): the bead's record, its
// neighbours' places and its part of the Philox rounds are set up once a block.
// DEG: the most bonds of a bead (a loop of bonds that ends early would keep the
// compiler from placing loads and Philox rounds side by side).
//
// 2.0M beads in combs of 40 (a backbone of 24, eight side chains of two): 25.1 us a
// sweep in k_run, where k_sweep (a block a tile, every trial exact) took 77.6.  Of
// these 6 us are barriers and the field, 5 the exact trials (5.8 % of all: the ends
// of the side chains have one bond and pass the screen five times as often), the
// rest the screen, whose twelve scattered reads of shared memory a trial cost it
// twice the linear one's time.  One row of trials a step 29.1 us, with the places
// computed anew each step 31; a bit mask a lane instead of the list 25.6.
template <int DEG, int FORM, int KEYS>
__device__ __forceinline__ unsigned graph_tile(typename SweepLayout<FORM>::Warp* wp, const SweepSys& c, const SweepConsts& s,
                                               const TileRef& t, int n_chains, const ArchDev* A, bool screened,
                                               const PhiloxKeys& keys, const float4* ntab) {
    constexpr int kStride = SweepLayout<FORM>::kStride;
    const int lane = threadIdx.x & 31;
    const uint32_t tab = screen_lane();
    const int n_colors = A->n_colors;
    unsigned nacc = 0;
#pragma unroll 1
    for (int k = 0; k < n_colors; ++k) {
        const GraphBead* const beads = A->graph + A->color_off[k];
        const int n = A->color_off[k + 1] - A->color_off[k], width = A->color_width[k], per = A->color_per[k];
        const uint32_t magic = A->color_magic[k];
        int slot0 = 0, c0 = 0;
#pragma unroll 1
        do {
            int have = 0;
            if (!screened) {
                have = n_chains * n;
                slot0 = n;
            }
#pragma unroll 1
            while (slot0 < n) {
                const float* Q[2];
                int nbr[2][DEG], chain[2], item[2];
                float2 ab[2];
                uint64_t p0[2];
                const uint64_t m1s = (uint64_t)0xCD9E8D57u * s.step;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int at = lane + 32 * i, ci = at / width, slot = slot0 + at - ci * width;
                    const bool ok = ci < per && slot < n;
                    const GraphRec rec = graph_rec(beads, ok ? slot : 0);
                    chain[i] = ok ? c0 + ci : n_chains;  // none
                    item[i] = chain[i] * n + slot;
                    Q[i] = t.X + (chain[i] * s.L + (int)rec.bead());
                    ab[i] = *reinterpret_cast<const float2*>(&wp->by_deg[rec.deg()]);
#pragma unroll
                    for (int d = 0; d < DEG; ++d) nbr[i][d] = rec.nbr(d) - (int)rec.bead();
                    p0[i] = (uint64_t)0xD2511F53u * ((uint32_t)(m1s >> 32) ^ (KEYS == kKeysBoth ? keys.k[0] : s.k0) ^ rec.bead());
                }
                const f32x2 a2 = pack2(ab[0].x, ab[1].x), b2 = pack2(ab[0].y, ab[1].y), add = pack2(s.add, s.add);
                const f32x2 k2 = pack2(c.k2, c.k2), zero = pack2(0.0f, 0.0f);
                // full steps; a lane past the last chain looks at the tile's first bead
#pragma unroll 1
                for (; c0 < n_chains && have <= kListLen - 64; c0 += per) {
                    f32x2 f[3] = {zero, zero, zero};
                    const float *P[2], *O[2];
                    bool in[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        in[i] = chain[i] < n_chains;
                        P[i] = in[i] ? Q[i] : t.X;
                    }
                    const float x[2] = {P[0][0], P[1][0]}, y[2] = {P[0][kStride], P[1][kStride]},
                                z[2] = {P[0][2 * kStride], P[1][2 * kStride]};
#pragma unroll
                    for (int d = 0; d < DEG; ++d) {  // a missing bond is one with the bead itself
                        O[0] = in[0] ? P[0] + nbr[0][d] : t.X;
                        O[1] = in[1] ? P[1] + nbr[1][d] : t.X;
                        f[0] = fma2(pack2(__fsub_rn(O[0][0], x[0]), __fsub_rn(O[1][0], x[1])), k2, f[0]);
                        f[1] = fma2(pack2(__fsub_rn(O[0][kStride], y[0]), __fsub_rn(O[1][kStride], y[1])), k2, f[1]);
                        f[2] = fma2(pack2(__fsub_rn(O[0][2 * kStride], z[0]), __fsub_rn(O[1][2 * kStride], z[1])), k2, f[2]);
                    }
                    uint4 w[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        w[i] = bead_block<KEYS>(t.rng0 + (uint32_t)chain[i], (uint32_t)m1s, p0[i], s.k0, s.k1, keys);
                    const f32x2 vx = fma2(f[0], a2, pack2(screen_normal(w[0].x, tab), screen_normal(w[1].x, tab)));
                    const f32x2 vy = fma2(f[1], a2, pack2(screen_normal(w[0].y, tab), screen_normal(w[1].y, tab)));
                    const f32x2 vz = fma2(f[2], a2, pack2(screen_normal(w[0].z, tab), screen_normal(w[1].z, tab)));
                    const f32x2 q = fma2(vx, vx, fma2(vy, vy, mul2(vz, vz)));
                    const f32x2 u = pack2(__fmaf_rn(log2_below_u(accept_word(w[0])), s.u1, s.u0),
                                          __fmaf_rn(log2_below_u(accept_word(w[1])), s.u1, s.u0));
                    const f32x2 lim = fma2(b2, fma2(f[0], f[0], fma2(f[1], f[1], fma2(f[2], f[2], u))), add);
                    float qi[2], li[2];
                    unpack2(q, qi[0], qi[1]);
                    unpack2(lim, li[0], li[1]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const bool pass = !(qi[i] > li[i]) && in[i];  // NaN passes
                        const uint32_t who = __ballot_sync(0xffffffffu, pass);
                        if (pass) wp->list[have + __popc(who & ((1u << lane) - 1u))] = (uint16_t)item[i];
                        have += __popc(who);
                        chain[i] += per;
                        item[i] += per * n;
                        Q[i] += per * s.L;
                    }
                }
                if (c0 < n_chains) break;  // the list is full
                c0 = 0;
                slot0 += width;
            }
            __syncwarp();
#pragma unroll 1
            for (int r = lane; r < have; r += 32) {
                const int j = screened ? (int)wp->list[r] : r;
                const int cl = (int)div_magic((uint32_t)j, magic, n);
                const GraphRec rec = graph_rec(beads, j - cl * n);
                const float2 ca = *(reinterpret_cast<const float2*>(&wp->by_deg[rec.deg()]) + 1);
                const float* const first = t.X + cl * s.L;
                const float* const Q = first + rec.bead();
                Trial b;
                b.x = Q[0];
                b.y = Q[kStride];
                b.z = Q[2 * kStride];
                b.fx = b.fy = b.fz = 0.0f;
#pragma unroll
                for (int d = 0; d < DEG; ++d) {
                    const float* const O = first + rec.nbr(d);
                    add_bond(c.k2, b.x, b.y, b.z, O[0], O[kStride], O[2 * kStride], b.fx, b.fy, b.fz);
                }
                b.chain = t.rng0 + (uint32_t)cl;
                b.bead = rec.bead();
                b.typ = rec.type() * c.n_cells;
                b.p = cl * s.L + (int)rec.bead();
                b.cc = ca.x;
                b.ac4 = ca.y;
                nacc += settle<FORM, KEYS>(c, s, t, keys, ntab, b, true) ? 1u : 0u;
            }
            __syncwarp();
        } while (slot0 < n);
    }
    return nacc;
}

// A warp of a move kernel: its tile, its shared memory and the constants of the
// system and architecture it is at.  ONE: the launch has one system, whose
// constants are parameters (instruction operands).
template <bool ONE, int FORM, int KEYS>
struct Mover {
    using Lay = SweepLayout<FORM>;
    const SweepArgs& a;
    typename Lay::Warp* const wp;
    const float4* const ntab;
    const int lane;
    SweepConsts s;
    SysDev* S = nullptr;
    const ArchDev* A = nullptr;
    const uint8_t* types = nullptr;
    uint32_t rng_base = 0u, h_magic = 0u, parity = 0u;
    float span = 0.0f;
    int mode = 0;  // 0: the system's sweeps are done; 1: resolve every trial; 2: screen

    __device__ __forceinline__ Mover(const SweepArgs& args, unsigned char* smem)
        : a(args),
          wp(reinterpret_cast<typename Lay::Warp*>(smem + Lay::kTabBytes) + (threadIdx.x >> 5)),
          ntab(reinterpret_cast<const float4*>(smem)),
          lane(threadIdx.x & 31) {}
    __device__ __forceinline__ const SweepSys& sys() const { return ONE ? a.sys : wp->sys; }

    // One lane: has the buffer filled with a tile, from the 16-byte boundary below it.
    __device__ __forceinline__ void load(const WarpTile& t) {
        const SweepSys& c = ONE ? a.sys : t.sys->sweep;
        const uint32_t bar = smem_addr(&wp->full), dst = smem_addr(wp->pos + 4);
        const int off = (int)(t.bead0 & 3);
        const uint32_t bytes = (uint32_t)((off + t.n_beads + 3) & ~3) * 4u;
        const int64_t g = t.bead0 - off;
        mbar_expect(bar, 3u * bytes);
        bulk_load(dst, c.x + g, bytes, bar, a.once != 0);
        bulk_load(dst + 4u * Lay::kStride, c.y + g, bytes, bar, a.once != 0);
        bulk_load(dst + 8u * Lay::kStride, c.z + g, bytes, bar, a.once != 0);
    }

    // All threads of the block: the tables, the warp's barrier, and its first tile on
    // the way (as soon as the kernel before, if this one may begin beside it, is done).
    __device__ __forceinline__ void start(unsigned char* smem, const WarpTile& t, bool any) {
        if (lane == 0) {
            mbar_init(smem_addr(&wp->full));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        wp->moved[lane] = 0u;
        float4* tab = reinterpret_cast<float4*>(smem);
        for (int i = threadIdx.x; i < SCMF_NORMAL_SEGS; i += blockDim.x) tab[i] = __ldg(normal_table() + i);
        float2* screen = reinterpret_cast<float2*>(smem + kScreenTabAt);
        if (FORM != kFormUnscreened)
            for (int i = threadIdx.x; i < SCMF_SCREEN_SEGS * kScreenCopies; i += blockDim.x)
                screen[i] = __ldg(screen_table() + i / kScreenCopies);
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        if (lane == 0) {
            fence_async();
            if (any) load(t);
        }
        __syncthreads();
    }

    // Turns to a tile's architecture (what no sweep changes of it); set() has the rest.
    __device__ __forceinline__ void turn_to(const WarpTile& t) {
        if (!ONE && t.sys != S) {
            __syncwarp();
            const uint32_t* src = reinterpret_cast<const uint32_t*>(&t.sys->sweep);
            for (int i = lane; i < (int)(sizeof(SweepSys) / 4); i += 32) reinterpret_cast<uint32_t*>(&wp->sys)[i] = src[i];
            __syncwarp();
        }
        if (FORM == kFormGraph && t.sys != S) {
            __syncwarp();
            if (lane <= kGraphDeg) wp->by_deg[lane] = t.sys->by_deg[lane];
            __syncwarp();
        }
        S = t.sys;
        A = t.arch;
        types = A->types;
        rng_base = (uint32_t)A->rng_base;
        h_magic = A->tpc_magic;
    }

    // The constants of a sweep of chains of L beads.  `done`: sweeps of the system made
    // before this one; omega_span: its omega's.
    __device__ __forceinline__ void set(int L, uint32_t done, bool active, float omega_span) {
        const SweepSys& c = sys();
        span = omega_span;
        s.L = L;
        s.h = (L + 1) >> 1;
        s.h_magic = h_magic;
        s.step = done + 1u;
        s.k0 = c.seed_lo;
        s.k1 = c.seed_hi;
        s.k2 = c.k2;
        s.a1 = c.screen.a[1];
        s.a2 = c.screen.a[2];
        s.b1 = c.screen.b[1];
        s.b2 = c.screen.b[2];
        s.add = c.screen.add;
        s.u0 = __fmul_rn(c.screen.u, __fadd_rn(span, 0x1p-18f));
        s.u1 = __fmul_rn(c.screen.u, -0x1.62e7p-1f);  // a little over ln 2
        const bool screened = FORM != kFormUnscreened && c.screen.on >= (FORM == kFormGraph ? kScreenGraphs : kScreenTiles);
        mode = !active ? 0 : screened && s.L > 1 ? 2 : 1;  // one bead has no energy to screen by
        const int k = lane & (s.h - 1);
        s.pc = pair_consts(s, k == 0, false, k == s.h - 1);
        s.head = pair_head<KEYS>(2u * (uint32_t)k, s.step, s.k0, a.keys);
    }

    // Waits for the tile asked for; false (and the error word) if it does not come.
    __device__ __forceinline__ bool arrived() {
        const bool ok = mbar_wait(smem_addr(&wp->full), parity);
        if (!ok && lane == 0) atomicOr(&S->error_word, kErrorTile);
        parity ^= 1u;
        return ok;
    }

    __device__ __forceinline__ bool graph() const { return FORM == kFormGraph && A->graph; }

    // The trials of the tile in the buffer that may be accepted (screen_tile's masks).
    __device__ __forceinline__ void screen(const WarpTile& t, uint32_t& even, uint32_t& odd) {
        const int off = (int)(t.bead0 & 3);
        const uint32_t rng0 = rng_base + t.chain, tab = screen_lane();
        const float* X = wp->pos + 4 + off;
        even = odd = 0u;
        if (FORM != kFormUnscreened && mode == 2) {
            if ((s.L | off) & 1)
                screen_tile<2, FORM, KEYS>(s, X, rng0, t.n_chains, a.keys, tab, even, odd);
            else if (32 % s.h)
                screen_tile<1, FORM, KEYS>(s, X, rng0, t.n_chains, a.keys, tab, even, odd);
            else
                screen_tile<0, FORM, KEYS>(s, X, rng0, t.n_chains, a.keys, tab, even, odd);
        } else if (mode == 1) {
            even = odd = row_mask(t.n_chains * s.h);
        }
    }
    // Makes them.  Returns the lane's accepted moves.
    __device__ __forceinline__ unsigned resolve(const WarpTile& t, uint32_t even, uint32_t odd, bool write) {
        TileRef ref{wp->pos + 4 + (int)(t.bead0 & 3), t.bead0, rng_base + t.chain, t.n_chains * s.h, types, span,
                    a.move_counts != 0, write};
        if (graph()) {
            if (mode == 0) return 0u;
            return A->max_deg <= 3 ? graph_tile<3, FORM, KEYS>(wp, sys(), s, ref, t.n_chains, A, mode == 2, a.keys, ntab)
                                   : graph_tile<kGraphDeg, FORM, KEYS>(wp, sys(), s, ref, t.n_chains, A, mode == 2, a.keys, ntab);
        }
        return resolve_tile<FORM, KEYS>(wp, sys(), s, ref, a.keys, ntab, even, odd);
    }
    // One sweep of the tile.
    __device__ __forceinline__ unsigned move(const WarpTile& t, bool write) {
        uint32_t even = 0u, odd = 0u;
        if (!graph()) screen(t, even, odd);
        return resolve(t, even, odd, write);
    }
};

// Tile i of a launch: from the list, or where the launch has one system by
// counting (each architecture's chains in tiles of `per`).
template <bool ONE>
__device__ __forceinline__ WarpTile tile_at(const SweepArgs& a, int i) {
    if (!ONE) return a.tiles[i];
    int k = 0;
    while (k + 1 < a.n_arch && i >= a.arch[k + 1].first) ++k;
    const SweepArch& r = a.arch[k];
    const int chain = (i - r.first) * r.per;
    WarpTile t;
    t.sys = a.system;
    t.arch = r.arch;
    t.bead0 = r.bead_base + (int64_t)chain * r.length;
    t.chain = (uint32_t)chain;
    t.n_chains = min(r.per, r.n_chains - chain);
    t.n_beads = t.n_chains * r.length;
    t.length = r.length;
    return t;
}

// One move of the systems of a launch.  One CTA per SM; each warp strides over
// the tiles (whole chains of one architecture, up to SweepLayout::kBeads beads), whose
// positions come by bulk copies, the next tile's from the moment the current one
// is done.  Beads that move are written back, and nothing else.
//
// Warps that make equal tiles in step would ask for their positions together and
// then leave memory idle together.  Where a warp makes several tiles, it begins
// with a quarter, a half, three quarters or all of its first one (by its place
// among the four warps of its SM sub-partition) and ends with the rest: 0.322 ->
// 0.313 ms on the large system.
//
// A chained launch (LaunchShape::chained) reads only what no sweep changes before
// griddepcontrol.wait in start().
template <bool ONE, int FORM, int KEYS>
__global__ void __launch_bounds__(SweepLayout<FORM>::kWarps * 32, 1) k_sweep_warp(const __grid_constant__ SweepArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Mover<ONE, FORM, KEYS> m(a, smem_raw);
    // consecutive tiles go to different SMs, so that few tiles spread over all of them
    const int warp = (int)(threadIdx.x >> 5), nwarps = (int)(blockDim.x >> 5);
    const int first = warp * (int)gridDim.x + (int)blockIdx.x, stride = nwarps * (int)gridDim.x;
    const int turns = first < a.n_tiles ? (a.n_tiles - first + stride - 1) / stride : 0;
    WarpTile t{};
    if (turns > 0) t = tile_at<ONE>(a, first);
    const WarpTile whole = t;
    const int begin = turns >= 4 ? max(1, t.n_chains * (4 * warp / nwarps + 1) / 4) : t.n_chains;  // chains of the first part
    const int parts = turns + (begin < whole.n_chains ? 1 : 0);
    t.n_chains = begin;
    t.n_beads = begin * t.length;
    if (turns > 0) m.turn_to(t);  // may run beside the field step before (start)
    m.start(smem_raw, t, turns > 0);
#pragma unroll 1
    for (int q = 0; q < parts; ++q) {
        WarpTile next = whole;
        if (q + 1 < turns) {
            next = tile_at<ONE>(a, first + (q + 1) * stride);
        } else {
            next.chain += (uint32_t)begin;
            next.bead0 += (int64_t)begin * next.length;
            next.n_chains -= begin;
            next.n_beads -= begin * next.length;
        }
        if (q == 0 || t.arch != m.A) {
            const uint32_t step = t.sys->step, stop = t.sys->stop_step;
            const float omega_span = t.sys->omega_span;
            if (q) m.turn_to(t);
            m.set(t.length, step, step < stop, omega_span);
        }
        if (!m.arrived()) return;
        unsigned nacc = m.move(t, true);
        fence_async();  // this lane's reads and writes of the buffer, before the next copies land
        __syncwarp();
        if (q + 1 < parts && m.lane == 0) m.load(next);
        if (__any_sync(0xffffffffu, nacc)) {
            nacc = warp_sum(nacc);
            if (m.lane == 0) atomicAdd(&m.S->slot_acc[(first + q) % kSlots], (unsigned long long)nacc);
        }
        t = next;
    }
}

// ------------------------------------------------- every trial, in registers
// One move of systems that are not screened, of linear chains of up to 64 beads: a row of
// lanes has whole chains, each lane a bead pair in registers.  It makes the even bead and
// then the odd one, with neighbours by shuffles, and loads the next row's pair meanwhile.
// Nothing of a trial is left out, so there is nothing to gather and no reason to keep a
// tile: without its buffers an SM has 24 warps, and room for copies of the normal table
// (lane l reads copy l mod 8, so the eight lanes of a 16-byte phase never meet in a bank).
// Bound by instruction issue, with the latency of omega's
// reads behind it.  These may go through L1: omega does not change while the kernel
// runs, and the old and the new cell of a small step share a line.
//
// A sweep of 20.5M beads in chains of 32, nine trials in ten accepted: 223 us on 128^3
// cells and 229 on 96^3, where tiles in shared memory took 379 and 392 (four warps a
// scheduler do not cover the latency of an exact trial, and each move was three
// scattered words to memory); 20M single beads 349 and 527; 20 systems of 4.7M beads 77
// and 117.  With 28 warps and one copy of the normal table in tiles of 640 beads 318.
// Without the prefetch of the next row 249, the Philox blocks of a pair made apart 237.
//
// ONE: one system of chains of even lengths, whose pairs lie on 8-byte boundaries.
// FOLD: SweepSys::fold of the one system, or 3: each system's own.
constexpr int kPairCopies = 8;
template <bool ONE>
constexpr int pairs_smem() {
    return SCMF_NORMAL_SEGS * kPairCopies * (int)sizeof(float4) + (ONE ? 0 : kSweepForms[kFormPairsList].warps * (int)sizeof(SweepSys));
}

template <int FOLD>
__device__ __forceinline__ int cell_of_fold(const SweepSys& c, float x, float y, float z) {
    if (FOLD == 0)
        return fold_pow2(x, c.inv_d[0], c.n[0] - 1) +
               c.n[0] * (fold_pow2(y, c.inv_d[1], c.n[1] - 1) + c.n[1] * fold_pow2(z, c.inv_d[2], c.n[2] - 1));
    if (FOLD == 1)
        return fold_magic(x, c.inv_d[0], c.n[0], c.fold_off[0], c.fold_mag[0]) +
               c.n[0] * (fold_magic(y, c.inv_d[1], c.n[1], c.fold_off[1], c.fold_mag[1]) +
                         c.n[1] * fold_magic(z, c.inv_d[2], c.n[2], c.fold_off[2], c.fold_mag[2]));
    if (FOLD == 2)
        return fold(x, c.inv_d[0], c.n[0]) +
               c.n[0] * (fold(y, c.inv_d[1], c.n[1]) + c.n[1] * fold(z, c.inv_d[2], c.n[2]));
    return cell_index(c, x, y, z);
}

// A lane's trial (where act) with trial_f's expressions, under branches that the warp
// takes as one; a bead that moves has its new position afterwards.
template <int FOLD>
__device__ __forceinline__ bool trial_pair(const SweepSys& c, float& x, float& y, float& z, float fx, float fy, float fz,
                                           float cc, float ac4, float n0, float n1, float n2, uint32_t aw, float span,
                                           bool act, uint32_t typ, int& c_old, int& c_new) {
    const float dx = __fmaf_rn(c.A, fx, __fmul_rn(c.R, n0));
    const float dy = __fmaf_rn(c.A, fy, __fmul_rn(c.R, n1));
    const float dz = __fmaf_rn(c.A, fz, __fmul_rn(c.R, n2));
    const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
    const float fd = __fmaf_rn(fx, dx, __fmaf_rn(fy, dy, __fmul_rn(fz, dz)));
    const float deb = __fmul_rn(ac4, __fmaf_rn(cc, d2, __fmul_rn(-2.0f, fd)));
    const float u = u01(aw);
    c_old = c_new = 0;
    bool acc = false;
    if (__any_sync(0xffffffffu, act && maybe_accepted(deb, span, log_lower(u)))) {
        const float px = __fadd_rn(x, dx), py = __fadd_rn(y, dy), pz = __fadd_rn(z, dz);
        c_old = cell_of_fold<FOLD>(c, x, y, z);
        c_new = cell_of_fold<FOLD>(c, px, py, pz);
        const float dE = __fadd_rn(__fsub_rn(c.omega[typ + c_new], c.omega[typ + c_old]), deb);
        // log_lower decides without the logarithm for the rejected ones (trial_f)
        acc = dE < 0.0f;
        const bool near = !acc && -dE > log_lower(u);
        if (__any_sync(0xffffffffu, near)) acc = acc || (near && log_f(u) < -dE);
        acc = acc && act;
        if (acc) {
            x = px;
            y = py;
            z = pz;
        }
    }
    return acc;
}

template <bool ONE, int FOLD, int KEYS>
__global__ void __launch_bounds__(kSweepForms[ONE ? kFormPairs : kFormPairsList].warps * 32, 1)
    k_sweep_pairs(const __grid_constant__ SweepArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    float4* const table = reinterpret_cast<float4*>(smem_raw);
    for (int i = threadIdx.x; i < SCMF_NORMAL_SEGS * kPairCopies; i += blockDim.x) table[i] = __ldg(normal_table() + i / kPairCopies);
    const float4* const ntab = table + (lane & (kPairCopies - 1));
    SweepSys* const own = reinterpret_cast<SweepSys*>(table + SCMF_NORMAL_SEGS * kPairCopies) + warp;  // !ONE
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncthreads();
    const int first = warp * (int)gridDim.x + (int)blockIdx.x, stride = nwarps * (int)gridDim.x;
    const SweepSys& c = ONE ? a.sys : *own;
    SysDev* S = nullptr;
    const ArchDev* A = nullptr;
    uint32_t step = 0u, stop = 0u, rng0 = 0u, typ_e = 0u, typ_o = 0u;
    float span = 0.0f, cc_e = 0.0f, ac_e = 0.0f, cc_o = 0.0f, ac_o = 0.0f, k2l = 0.0f, k2o = 0.0f, k2r = 0.0f;
    int slot = 0, k = 0, per = 1;
    PairHead head{};
    unsigned nacc = 0;
    const auto flush = [&](int at) {  // the system's accepted moves so far
        nacc = warp_sum(nacc);
        if (lane == 0 && nacc) atomicAdd(&S->slot_acc[at % kSlots], (unsigned long long)nacc);
        nacc = 0u;
    };
#pragma unroll 1
    for (int i = first; i < a.n_tiles; i += stride) {
        const WarpTile t = tile_at<ONE>(a, i);
        const int L = t.length;
        if (t.arch != A) {
            if (t.sys != S) {
                if (!ONE && S) flush(i);
                S = t.sys;
                if (!ONE) {
                    __syncwarp();
                    const uint32_t* src = reinterpret_cast<const uint32_t*>(&S->sweep);
                    for (int w = lane; w < (int)(sizeof(SweepSys) / 4); w += 32) reinterpret_cast<uint32_t*>(own)[w] = src[w];
                    __syncwarp();
                }
                step = S->step + 1u;
                stop = S->stop_step;
                span = S->omega_span;
            }
            A = t.arch;
            const int h = (L + 1) >> 1;
            per = 32 / h;
            slot = (int)div_magic((uint32_t)lane, A->tpc_magic, h);
            k = lane - slot * h;
            rng0 = (uint32_t)A->rng_base;
            const bool has_l = k > 0, has_o = ONE || 2 * k + 1 < L, has_r = 2 * k + 2 < L;
            k2l = has_l ? c.k2 : 0.0f;
            k2o = has_o ? c.k2 : 0.0f;
            k2r = has_r ? c.k2 : 0.0f;
            const int deg = (has_l ? 1 : 0) + (has_o ? 1 : 0);
            cc_e = deg == 2 ? c.cdeg[2] : deg == 1 ? c.cdeg[1] : 0.0f;
            ac_e = deg == 2 ? c.ac4[2] : deg == 1 ? c.ac4[1] : 0.0f;
            cc_o = has_r ? c.cdeg[2] : c.cdeg[1];
            ac_o = has_r ? c.ac4[2] : c.ac4[1];
            typ_e = (uint32_t)__ldg(A->types + 2 * k) * c.n_cells;
            typ_o = has_o ? (uint32_t)__ldg(A->types + 2 * k + 1) * c.n_cells : 0u;
            head = pair_head<KEYS>(2u * (uint32_t)k, step, c.seed_lo, a.keys);
        }
        if (step > stop) continue;  // the system's sweeps are done
        const bool has_o = ONE || 2 * k + 1 < L, aligned = ONE || ((L | (int)t.bead0) & 1) == 0;
        float* const X = c.x + t.bead0;
        float* const Y = c.y + t.bead0;
        float* const Z = c.z + t.bead0;
        float nx[2], ny[2], nz[2];  // the next row's pair
        const auto fetch = [&](int c0) {
            const int p = min(c0 + slot, t.n_chains - 1) * L + 2 * k;
            if (aligned) {
                const float2 x = __ldcs(reinterpret_cast<const float2*>(X + p)), y = __ldcs(reinterpret_cast<const float2*>(Y + p)),
                             z = __ldcs(reinterpret_cast<const float2*>(Z + p));
                nx[0] = x.x, nx[1] = x.y, ny[0] = y.x, ny[1] = y.y, nz[0] = z.x, nz[1] = z.y;
            } else {
                const int q = p + (has_o ? 1 : 0);
                nx[0] = __ldcs(X + p), ny[0] = __ldcs(Y + p), nz[0] = __ldcs(Z + p);
                nx[1] = __ldcs(X + q), ny[1] = __ldcs(Y + q), nz[1] = __ldcs(Z + q);
            }
        };
        fetch(0);
#pragma unroll 1
        for (int c0 = 0; c0 < t.n_chains; c0 += per) {
            const int cl = min(c0 + slot, t.n_chains - 1), p = cl * L + 2 * k;
            const bool act = slot < per && c0 + slot < t.n_chains;
            float xe = nx[0], xo = nx[1], ye = ny[0], yo = ny[1], ze = nz[0], zo = nz[1];
            if (c0 + per < t.n_chains) fetch(c0 + per);
            // the odd bead before, or where there is none the bead itself, and no spring
            float lx = __shfl_up_sync(0xffffffffu, xo, 1), ly = __shfl_up_sync(0xffffffffu, yo, 1), lz = __shfl_up_sync(0xffffffffu, zo, 1);
            if (k == 0) lx = xe, ly = ye, lz = ze;
            uint4 we, wo;
            pair_blocks<KEYS>(rng0 + t.chain + (uint32_t)cl, head, c.seed_lo, c.seed_hi, a.keys, we, wo);
            float n0, n1, n2, fx = 0.0f, fy = 0.0f, fz = 0.0f;
            int old_e, new_e, old_o = 0, new_o = 0;
            normals3<kPairCopies>(we, ntab, n0, n1, n2);
            add_bond(k2l, xe, ye, ze, lx, ly, lz, fx, fy, fz);
            add_bond(k2o, xe, ye, ze, xo, yo, zo, fx, fy, fz);
            const bool me = trial_pair<FOLD>(c, xe, ye, ze, fx, fy, fz, cc_e, ac_e, n0, n1, n2, accept_word(we), span, act, typ_e, old_e, new_e);
            bool mo = false;
            if (ONE || L > 1) {
                // the even bead after, moved
                float rx = __shfl_down_sync(0xffffffffu, xe, 1), ry = __shfl_down_sync(0xffffffffu, ye, 1), rz = __shfl_down_sync(0xffffffffu, ze, 1);
                if (2 * k + 2 >= L) rx = xo, ry = yo, rz = zo;
                normals3<kPairCopies>(wo, ntab, n0, n1, n2);
                fx = fy = fz = 0.0f;
                add_bond(c.k2, xo, yo, zo, xe, ye, ze, fx, fy, fz);
                add_bond(k2r, xo, yo, zo, rx, ry, rz, fx, fy, fz);
                mo = trial_pair<FOLD>(c, xo, yo, zo, fx, fy, fz, cc_o, ac_o, n0, n1, n2, accept_word(wo), span, act && has_o, typ_o, old_o, new_o);
            }
            nacc += (me ? 1u : 0u) + (mo ? 1u : 0u);
            const bool count_e = me && new_e != old_e, count_o = mo && new_o != old_o;
            if (a.move_counts && __any_sync(0xffffffffu, count_e || count_o)) {
                if (count_e) count_move(c.counts, c.count16 != 0, typ_e, old_e, new_e);
                if (count_o) count_move(c.counts, c.count16 != 0, typ_o, old_o, new_o);
            }
            if (aligned) {
                if (act) {
                    __stcs(reinterpret_cast<float2*>(X + p), make_float2(xe, xo));
                    __stcs(reinterpret_cast<float2*>(Y + p), make_float2(ye, yo));
                    __stcs(reinterpret_cast<float2*>(Z + p), make_float2(ze, zo));
                }
            } else {
                if (me) X[p] = xe, Y[p] = ye, Z[p] = ze;
                if (mo) X[p + 1] = xo, Y[p + 1] = yo, Z[p + 1] = zo;
            }
        }
    }
    if (S) flush(first);
}

// ------------------------------------------------------ many sweeps a launch
// A barrier of all CTAs of a (cooperative) launch, on a count in global memory
// that only grows, by one a CTA and barrier.  CTAs that give up do so after different
// numbers of barriers: from then on the barrier is broken, and no launch uses it again.
struct GridBarrier {
    const RunArgs& r;           // barrier: the count, and after it a word that is set when the barrier breaks
    unsigned long long target;  // thread 0's
    // The count is a whole number of barriers until the last CTA comes to the first one.
    // Thread 0 says in *s_ok whether the barrier is whole.
    __device__ __forceinline__ GridBarrier(const RunArgs& run, int* s_ok) : r(run), target(0) {
        if (threadIdx.x == 0) {
            target = __ldcg(r.barrier) / gridDim.x * gridDim.x;
            *s_ok = __ldcg(r.barrier + 1) == 0ull;
        }
    }
    __device__ __forceinline__ void arrive() {
        __syncthreads();
        if (threadIdx.x == 0) {
            target += gridDim.x;
            asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(r.barrier) : "memory");
        }
    }
    // False (to all threads of the CTA) after r.wait.  Thread 0 calls `then` before the
    // others go on.
    template <typename Then>
    __device__ __forceinline__ bool wait(int* s_ok, const Then& then) {
        if (threadIdx.x == 0) {
            unsigned long long now;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(r.barrier) : "memory");
            if (now < target) {
                const long long t0 = clock64();
                do {
                    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(r.barrier) : "memory");
                } while (now < target && (uint32_t)((clock64() - t0) >> kWaitShift) < r.wait);
            }
            *s_ok = now >= target;
            then();
        }
        __syncthreads();
        return *s_ok != 0;
    }
};

// Whether sweep `step` ends with a field update (test.cpp:42).
__device__ __forceinline__ bool updates_field(int rule, uint32_t step) { return rule == 1 || step % 10u != 0u; }

// The screen of the next sweep runs before its omega is known, for spans up to
// this times the last one (the span moves by the omega of a bead or two in a few
// cells); with more, the sweep is screened again.
constexpr float kSpanAhead = 1.125f;

// The omega span that the sweep after `done` sweeps uses, in a launch that
// started at `base`: of the last field update, from the launch's slots (om_keys,
// by the update's step mod 3) or, before its first one, the system's.
__device__ __forceinline__ float span_after(const SysDev* S, int rule, uint32_t done, uint32_t base) {
    const uint32_t at = updates_field(rule, done) ? done : done - 1u;
    if (done == base || at == base) return __ldcg(&S->omega_span);
    const uint32_t kx = __ldcg(&S->om_keys[at % 3u][0]), kn = __ldcg(&S->om_keys[at % 3u][1]);
    const float span = kx >= kn ? __fsub_rn(ord_val(kx), ord_val(kn)) : INFINITY;
    return span >= 0.0f ? span : INFINITY;  // NaN (inf - inf): no bound
}

// The warp's largest and smallest omega into a pair of ordered keys.
__device__ __forceinline__ void fold_span(uint32_t* keys, float wmax, float wmin) {
    const uint32_t kx = __reduce_max_sync(0xffffffffu, ord_key(wmax)), kn = __reduce_min_sync(0xffffffffu, ord_key(wmin));
    if ((threadIdx.x & 31) == 0 && kx >= kn) {  // the warp saw a non-NaN omega
        atomicMax(keys, kx);
        atomicMin(keys + 1, kn);
    }
}

// The step at which a system stops: it goes no further once a wait has run out on it,
// when its counts have moved and its positions may not have been written.
__device__ __forceinline__ uint32_t stop_of(const SysDev* S) {
    const uint32_t word = S->error_word, stop = S->stop_step;
    return word & (kErrorTile | kErrorBarrier) ? 0u : stop;
}

// Closes a system after its sweeps of a launch (one block).
__device__ __forceinline__ void close_run(const RunSystem& rs, const RunArgs& r, unsigned long long* s_acc, double* s_ef) {
    SysDev* S = rs.sys;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const uint32_t base = S->step, left = S->run_stop > base ? S->run_stop - base : 0u;
    const uint32_t made = min((uint32_t)r.n_sweeps, left);
    if (made) {  // block-uniform
        unsigned long long all = 0, last = 0;
        for (int i = tid; i < kSlots; i += blockDim.x) {
            all += __ldcg(&S->slot_acc[i]);
            last += __ldcg(&S->slot_last[i]);
            S->slot_acc[i] = 0ull;
            S->slot_last[i] = 0ull;
        }
        double f = 0.0;
        for (int i = tid; i < rs.field_count; i += blockDim.x) f += __ldcg(r.ef_part + rs.field_first + i);
        all = warp_sum(all);
        last = warp_sum(last);
        f = warp_sum(f);
        if (lane == 0) {
            s_acc[warp] = all;
            s_acc[32 + warp] = last;
            s_ef[warp] = f;
        }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < nwarps; ++w) {
                all += s_acc[w];
                last += s_acc[32 + w];
                f += s_ef[w];
            }
            const uint32_t step = base + made;
            S->last_accepts = last;
            S->total_accepts += all;
            S->total_moves += (unsigned long long)made * (unsigned long long)S->n_beads;
            S->e_field = f;
            if (S->avg && S->avg_every) S->avg_samples += step / S->avg_every - base / S->avg_every;
            S->omega_span = span_after(S, S->field_rule, step, base);
            S->step = step;
        }
    }
    __syncthreads();
}

// A launch whose blocks did not come to a barrier: the error word of every system.
__device__ __forceinline__ void give_up(const RunArgs& r) {
    if (threadIdx.x == 0) {
        for (int i = 0; i < r.n_sys; ++i) atomicOr(&r.systems[i].sys->error_word, kErrorBarrier);
        atomicExch(r.barrier + 1, 1ull);
    }
}

// A warp's field step over one tile of cells of N types (0: any number): omega
// of the new counts, and the averaging sample where the sweep takes one.  Returns
// the lane's field energy, where it is asked for.
template <int N>
__device__ __forceinline__ double field_tile_of(const FieldSys& f, int64_t cell0, int n_cells, bool upd, unsigned long long* avg,
                                                bool energy, float& wmax, float& wmin) {
    const int lane = threadIdx.x & 31;
    const int64_t NC = f.n_cells, end = cell0 + n_cells;
    const bool lit = f.literal != 0, c16 = f.count16 != 0;
    double ef = 0.0;
    if (N > 0 && !c16 && ((NC | cell0 | n_cells) & 3) == 0 && n_cells > 32) {
        for (int64_t cell = cell0 + 4 * lane; cell < end; cell += 128)
            ef += field_cells4<(N > 0 ? N : 1), true>(cell, NC, f.scale, lit, upd, f.counts, f.omega, f.cf, avg, wmax, wmin, energy);
    } else {
        for (int64_t cell = cell0 + lane; cell < end; cell += 32)
            ef += field_cell<N, true>(f.n_types, cell, NC, f.scale, lit, upd, c16, f.counts, f.omega, f.cf, avg, wmax, wmin, energy);
    }
    return ef;
}
__device__ __forceinline__ double field_tile(const FieldSys& f, int64_t cell0, int n_cells, bool upd, bool sample, bool energy,
                                             float& wmax, float& wmin) {
    unsigned long long* avg = sample ? f.avg : nullptr;
    switch (f.n_types) {
        case 1: return field_tile_of<1>(f, cell0, n_cells, upd, avg, energy, wmax, wmin);
        case 2: return field_tile_of<2>(f, cell0, n_cells, upd, avg, energy, wmax, wmin);
        case 3: return field_tile_of<3>(f, cell0, n_cells, upd, avg, energy, wmax, wmin);
        default: return field_tile_of<0>(f, cell0, n_cells, upd, avg, energy, wmax, wmin);
    }
}

// n_sweeps whole sweeps (move, field, statistics) of the systems of a launch in
// one cooperative launch, where every warp has one tile at most: its positions
// stay in shared memory from sweep to sweep, the tables and constants are set up
// once, and two grid barriers a sweep take the place of two kernel launches.  A
// sweep of such a system is mostly latency (launches, tables, descriptors, each
// a dependent trip to L2).  A sweep in this form against two kernels replayed
// from a graph: 32,000 beads 7.1 us against 18.6 us; 409,600 beads, unscreened,
// 12.5 against 22.7 us; 2.0M beads in chains of 33 18.8 against 28.9 us.  (Before
// the kernels of this file: 14.6, 20.7 and 55.4 us.)
//
// A screen needs nothing of the sweep before but the positions of its own tile and a
// bound on omega's span.  So the next sweep's screen runs between arriving at the
// barrier after the move and waiting there, with a span that is an eighth larger
// than the last one; the exact trials, after the field step, use the true one, and
// a sweep whose span is more than that is screened again.  Of the 7.1 us of 32,000
// beads the exact trials take 2.2, the screen 0.8, the field 1.5 and the barriers
// the rest (1.3 each at the least: arrival and a look at the count are a trip to L2
// each).  Screening after the field step took 8.2, with the field step's energy summed
// every sweep and each warp reading the span for itself 8.5.
template <bool ONE, int FORM, int KEYS>
__global__ void __launch_bounds__(SweepLayout<FORM>::kWarps * 32, 1)
    k_run(const __grid_constant__ SweepArgs a, const __grid_constant__ RunArgs r) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_ok;
    __shared__ float s_span;  // one system's, of the sweep to come
    __shared__ uint32_t s_keys[2];
    __shared__ unsigned long long s_acc[64];
    __shared__ double s_ef[32];
    auto* const wp = reinterpret_cast<typename SweepLayout<FORM>::Warp*>(smem_raw + SweepLayout<FORM>::kTabBytes) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const int first = (int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x, stride = (int)(blockDim.x >> 5) * (int)gridDim.x;
    const bool any = first < a.n_tiles;
    GridBarrier barrier(r, &s_ok);
    if (ONE && threadIdx.x == 0) s_span = a.system->omega_span;
    if (threadIdx.x < 2) s_keys[threadIdx.x] = threadIdx.x ? 0xFFFFFFFFu : 0u;
    for (int i = blockIdx.x; i < r.n_sys; i += gridDim.x) {  // the slot of the launch's first field step
        SysDev* S = r.systems[i].sys;
        const uint32_t step = S->step, stop = stop_of(S);
        if (threadIdx.x < 2) S->om_keys[(step + 1u) % 3u][threadIdx.x] = threadIdx.x ? 0xFFFFFFFFu : 0u;
        if (threadIdx.x == 0) S->run_stop = stop;  // for this block's close_run: other blocks may set the word meanwhile
    }
    {
        Mover<ONE, FORM, KEYS> m(a, smem_raw);
        WarpTile t{};
        if (any) t = tile_at<ONE>(a, first);
        m.start(smem_raw, t, any);
        if (any) {
            const uint32_t base = t.sys->step, stop = stop_of(t.sys);
            m.turn_to(t);
            const bool here = m.arrived();
            if (lane == 0) {
                wp->run.tile = t;
                wp->run.types = m.types;
                wp->run.rng_base = m.rng_base;
                wp->run.h_magic = m.h_magic;
                wp->run.base = base;
                wp->run.stop = stop;
                wp->run.rule = t.sys->field_rule;
                wp->run.active = here;
            }
            __syncwarp();
        }
    }
    if (!s_ok) return give_up(r);  // to be seen since the block's barrier in start()
    // the warp's field tile (its first, where it has several) and that one's system
    FieldSys* const fs = &wp->field;
    const auto at_field = [&](const FieldTile& t) {
        __syncwarp();
        const uint32_t* src = reinterpret_cast<const uint32_t*>(&t.sys->field);
        for (int i = lane; i < (int)(sizeof(FieldSys) / 4); i += 32) reinterpret_cast<uint32_t*>(fs)[i] = src[i];
        if (lane == 0) {
            fs->avg = t.sys->avg;
            fs->avg_every = t.sys->avg_every;
            wp->run.f_sys = t.sys;
            wp->run.cell0 = t.cell0;
            wp->run.n_cells = t.n_cells;
            wp->run.f_base = t.sys->step;
            wp->run.f_stop = stop_of(t.sys);
        }
        __syncwarp();
    };
    if (first < r.n_field) at_field(r.field[first]);
    unsigned acc_all = 0, acc_last = 0;  // of all the launch's sweeps, of the system's last
    uint32_t even = 0u, odd = 0u;        // the screen of the sweep to come, where it has been made,
    float screened_to = -INFINITY;       // which holds for spans up to this
    float span_now = INFINITY;           // the last sweep's span
#pragma unroll 1
    for (int sweep = 0; sweep < r.n_sweeps; ++sweep) {
        // pass 0: this sweep's move; pass 1: the screen of the next one, between arriving at the barrier and waiting
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            if (pass) barrier.arrive();
            if (!any || !wp->run.active || (pass && sweep + 1 == r.n_sweeps)) continue;
            const uint32_t base = wp->run.base, done = base + (uint32_t)(sweep + pass);
            if (done >= wp->run.stop) continue;
            Mover<ONE, FORM, KEYS> m(a, smem_raw);
            const WarpTile& t = wp->run.tile;
            m.S = t.sys;
            m.A = t.arch;
            m.types = wp->run.types;
            m.rng_base = wp->run.rng_base;
            float span;
            if (pass == 0) {
                span = ONE ? s_span : span_after(t.sys, wp->run.rule, done, base);
            } else {
                span = __fmul_rn(span_now, kSpanAhead);
                if (FORM == kFormUnscreened || !(span < INFINITY)) continue;
            }
            m.h_magic = wp->run.h_magic;
            m.set(t.length, done, true, span);
            const bool ahead = m.mode == 2 && !m.graph();  // a system whose screen may run ahead
            if (pass == 0 ? !m.graph() && !(span <= screened_to) : ahead) m.screen(t, even, odd);
            if (pass == 0) {
                acc_last = m.resolve(t, even, odd, false);
                acc_all += acc_last;
                span_now = span;
                screened_to = -INFINITY;
            } else if (ahead) {
                screened_to = span;
            }
        }
        if (!barrier.wait(&s_ok, [] {})) return give_up(r);
        float wmax = -INFINITY, wmin = INFINITY;
#pragma unroll 1
        for (int fi = first; fi < r.n_field; fi += stride) {
            if (r.n_field > stride) at_field(r.field[fi]);  // several field tiles a warp
            const uint32_t step = wp->run.f_base + (uint32_t)sweep + 1u, f_stop = wp->run.f_stop;
            if (step > f_stop) continue;
            const bool upd = updates_field(fs->rule, step), last = sweep + 1 == r.n_sweeps || step == f_stop;
            const bool sample = fs->avg && fs->avg_every && step % fs->avg_every == 0u;
            if (!upd && !last && !sample) continue;  // nothing to write and nothing to report
            if (!ONE) {
                wmax = -INFINITY;
                wmin = INFINITY;
            }
            double ef = field_tile(*fs, wp->run.cell0, wp->run.n_cells, upd, sample, last, wmax, wmin);
            if (last) {
                ef = warp_sum(ef);
                if (lane == 0) r.ef_part[fi] = ef;
            }
            if (!upd)
                wmax = -INFINITY, wmin = INFINITY;
            else if (!ONE)
                fold_span(wp->run.f_sys->om_keys[step % 3u], wmax, wmin);
        }
        if (ONE) {
            fold_span(s_keys, wmax, wmin);
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            if (ONE) {
                const uint32_t step = wp->run.base + (uint32_t)sweep + 1u;  // thread 0's warp has a tile
                if (s_keys[0]) {
                    atomicMax(&a.system->om_keys[step % 3u][0], s_keys[0]);
                    atomicMin(&a.system->om_keys[step % 3u][1], s_keys[1]);
                }
                s_keys[0] = 0u;
                s_keys[1] = 0xFFFFFFFFu;
                if (blockIdx.x == 0) {  // the slot of the next field step
                    a.system->om_keys[(step + 1u) % 3u][0] = 0u;
                    a.system->om_keys[(step + 1u) % 3u][1] = 0xFFFFFFFFu;
                }
            } else {
                for (int i = blockIdx.x; i < r.n_sys; i += gridDim.x) {
                    SysDev* S = r.systems[i].sys;
                    const uint32_t next = (S->step + (uint32_t)sweep + 2u) % 3u;
                    S->om_keys[next][0] = 0u;
                    S->om_keys[next][1] = 0xFFFFFFFFu;
                }
            }
        }
        if (sweep + 1 == r.n_sweeps && any) {
            const unsigned all = warp_sum(acc_all), last = warp_sum(acc_last);
            if (lane == 0) {
                SysDev* S = wp->run.tile.sys;
                if (all) atomicAdd(&S->slot_acc[first % kSlots], (unsigned long long)all);
                if (last) atomicAdd(&S->slot_last[first % kSlots], (unsigned long long)last);
            }
        }
        barrier.arrive();
        const bool ok = barrier.wait(&s_ok, [&] {
            if (ONE) s_span = span_after(a.system, wp->run.rule, wp->run.base + (uint32_t)sweep + 1u, wp->run.base);
        });
        if (!ok) return give_up(r);
    }
    if (any && wp->run.active) {  // the positions
        const SweepSys& c = ONE ? a.sys : wp->sys;
        const WarpTile& t = wp->run.tile;
        const float* P = wp->pos + 4 + (int)(t.bead0 & 3);
        for (int i = lane; i < t.n_beads; i += 32) {
            c.x[t.bead0 + i] = P[i];
            c.y[t.bead0 + i] = P[i + SweepLayout<FORM>::kStride];
            c.z[t.bead0 + i] = P[i + 2 * SweepLayout<FORM>::kStride];
        }
    }
    // the statistics of every system, in a fixed order
    for (int i = blockIdx.x; i < r.n_sys; i += gridDim.x) close_run(r.systems[i], r, s_acc, s_ef);
}

}  // namespace scmf
