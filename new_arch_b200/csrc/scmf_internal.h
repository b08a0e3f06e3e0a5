// Internal data model shared by the host engine (C++) and the kernels (CUDA).
//
// HBM layout of one system (all cudaMalloc'd, owned by the system):
//   x, y, z      float[n_beads]       SoA bead coordinates, unwrapped (the box is
//                                      folded only when a cell index is taken,
//                                      device_function.cu:313-360).  Beads of a
//                                      chain are contiguous; chains are grouped
//                                      by architecture (init_config.cu:610-629).
//   chain_id     uint32[n_chains]     storage slot -> global chain id (the first
//                                      Philox counter word).  Storage order is the id
//                                      order within each architecture (chain_id[chain_base
//                                      + c] = rng_base + c), which the kernels of warp tiles use to
//                                      compute the id instead of loading it; the other
//                                      kernels read this table.
//   counts[2]    uint32[n_types*n_cells] (or uint16 pairs)  per-type cell counts,
//                                      [type][z][y][x].  counts[cur] is kept the
//                                      grid of the positions: a fused sweep
//                                      moves a count for each accepted move that
//                                      leaves its cell.  The other buffer is
//                                      zero between calls (validation scratch).
//   omega        float[n_types*n_cells]  quasi-instantaneous field.
// plus a SysDev descriptor in device memory holding constants, the sweep
// counter and the statistics accumulators.
#pragma once
#include <stdint.h>

#include "scmf.h"

namespace scmf {

constexpr int kMaxTypes = 8;
constexpr int kMaxDeg = 8;
constexpr int kMaxColors = 8;
constexpr int kMaxLength = 4096;    // beads per chain (16-bit neighbour indices)
constexpr int kMaxTileBeads = 8192;  // beads staged in shared memory per tile
constexpr int kMaxWarps = 8;         // warps per move CTA (256 threads at most)
constexpr int kSlots = 32;           // spread of the accept-count atomics
constexpr uint32_t kInitStep = 0xFFFFFFFFu;

// Per-bead architecture record.
struct BeadInfo {
    uint8_t type, deg, color, pad;
    uint16_t nbr[kMaxDeg];
};

// A bead of an architecture that is no linear chain, as the move kernel of warp
// tiles reads it (in 16 bytes; the bonded beads in ascending order, the rest of
// `nbr` the bead itself).
constexpr int kGraphDeg = 6;
struct alignas(16) GraphBead {
    uint16_t bead;
    uint8_t deg, type;
    uint16_t nbr[kGraphDeg];
};

// Of the beads of some number of bonds: ScreenDev's a and b, c = 2k deg, A c / 4.
struct alignas(16) BondConsts {
    float a, b, c, ac4;
};

// One polymer architecture of one system.
struct ArchDev {
    const BeadInfo* beads;       // [length]
    const uint16_t* color_beads; // [length], beads grouped by colour
    const uint8_t* types;        // [length], monomer type per bead
    const GraphBead* graph;      // [length] in the order of color_beads; NULL for a linear chain
    int32_t length;
    int32_t n_colors;
    int32_t max_deg;
    int32_t color_off[kMaxColors + 1];
    uint32_t color_magic[kMaxColors];  // ceil(2^32 / n_in_colour): i / n == umulhi(i, magic)
    // graph: the screen's split of a colour, so that two rows of lanes have the same beads
    // from one step to the next: blocks of `width` beads, of `per` chains a step
    int32_t color_width[kMaxColors], color_per[kMaxColors];
    uint32_t len_magic;          // ceil(2^32 / length)
    uint32_t tpc_magic;          // magic of ceil(length / 2): bead pairs per chain
    int32_t n_chains;
    int32_t chain_base;          // first storage slot of this architecture in the system
    int32_t rng_base;            // random-stream id of its first chain: chain_base, or for a chain
                                 // shard the id that chain has in the whole system
    int64_t bead_base;           // first bead of this architecture in the system arrays
    float init_sigma;
};

// The screen of k_sweep_warp and k_run: constants of the test that proves a trial
// rejected before its exact normals, energy and omega are formed.
//
// With d = A f + R n the displacement and c = 2k deg, the energy that the trial
// kernels evaluate is, up to rounding,
//   dE_bond = (A c / 4)(c |d|^2 - 2 f.d) = (A c^2 R^2 / 4)|v|^2 - (A / 4)|f|^2,
//   v = n + ((A - 1/c) / R) f,
// and a trial is rejected when dE_bond >= span + L, span the largest fall of
// omega (SysDev::omega_span) and L >= -log u, because then dE = fl(fl(w_new -
// w_old) + dE_bond) >= max(0, -log u).  The screen has f exactly and n, hence v,
// to within delta in each component (SCMF_SCREEN_DELTA), and |v'|^2 <= (1 + eta)
// |v|^2 + (1 + 1/eta) 3 delta^2 for the v' it forms, so it rejects when
//   |v'|^2 > b (|f|^2 + (4 / A)(span + L)) + add
// with b = K / (c R)^2, K = (1 + eta)(1 + 2^-10), add = (1 + 1/eta) 3 delta^2
// and eta = 2^-6.  The 2^-10 and 2^-18 added to span + L cover every rounding on
// both sides (each a few 2^-24 of the terms bounded here).  v' is formed 2^30
// times as large and b, add 2^60 times, so that where a force is large enough to
// overflow the exact energy the right side is infinite and the trial passes.
// a and b are indexed by the bead's bonds.
struct ScreenDev {
    float a[3], b[3];  // a = (A - 1/c) / R
    float u;           // 4 / A
    float add;
    int32_t on;  // ScreenLevel (see screen_constants)
    int32_t pad;
};

// What the move kernels of warp tiles read of a system, fixed for its life.
struct SweepSys {
    float *x, *y, *z;
    const float* omega;
    uint32_t* counts;           // counts[0], which is always the current grid
    uint32_t n_cells;           // n_cells * n_types < 2^31
    float k2, A, R;
    float inv_d[3];
    int32_t n[3];
    int32_t fold;               // 0: every axis a power of two; 1: every axis of 2 to 256 cells; 2: others
    int32_t fold_off[3];        // fold_magic's
    uint32_t fold_mag[3];
    float cdeg[3], ac4[3];      // c = 2k deg and A c / 4
    uint32_t seed_lo, seed_hi;
    int32_t count16;
    ScreenDev screen;
};

// What the field step of k_run reads of a system.
struct FieldSys {
    const uint32_t* counts;
    float* omega;
    unsigned long long* avg;      // the averaging state as the launch finds it
    int64_t n_cells;
    float scale;
    int32_t n_types, literal, count16, rule;
    uint32_t avg_every;
    float cf[kMaxTypes * kMaxTypes];
};

struct SysDev {
    float* x;
    float* y;
    float* z;
    uint32_t* chain_id;
    uint32_t* counts[2];
    float* omega;
    int64_t n_cells;
    int64_t n_beads;
    int32_t n_types, nx, ny, nz;
    float inv_dx, inv_dy, inv_dz, scale;
    float lx, ly, lz;
    float k, k2, A, R;
    float cdeg[kMaxDeg + 1];    // c = 2k deg
    float ac4deg[kMaxDeg + 1];  // A c / 4
    float cf[kMaxTypes * kMaxTypes];
    int32_t hamiltonian, field_rule, count16, n_arch;
    uint32_t seed_lo, seed_hi;
    // mutable state
    uint32_t step;        // completed sweeps
    uint32_t cur;         // counts[cur] holds the counts of the current positions
    uint32_t error_word;
    uint32_t pad0;
    unsigned long long slot_acc[kSlots];  // accepted moves of the running sweep, cleared by k_close
    // statistics of the last completed sweep
    unsigned long long last_accepts, total_accepts, total_moves;
    double e_bond, e_field;
    uint32_t e_bond_step;  // step at which e_bond was last computed (+1; 0 = never)
    uint32_t pad1;
    // time-averaged density (io.cpp:57-94): the fused sweep adds the new counts
    // into avg at every sweep s with s % avg_every == 0 (avg NULL = off)
    unsigned long long* avg;         // [n_types * n_cells]
    unsigned long long avg_samples;  // sweeps accumulated
    uint32_t avg_every;
    uint32_t field_done;  // field tiles of the running launch finished (the last one closes the sweep)
    // fused sweeps leave the system alone once step reaches stop_step (the
    // served form gives each request its own sweep count inside a shared
    // round); 0xFFFFFFFF everywhere else
    uint32_t stop_step;
    uint32_t run_stop;  // stop_step as a launch of many sweeps found it, 0 for a system with an error word
    // counts the field step reads: NULL means counts[cur] (the grid of this
    // system's own beads); a chain shard points it at the sum over all shards
    const uint32_t* field_counts;
    // the span of omega: every field step folds the largest and smallest
    // non-NaN omega of its cells into om_max_key / om_min_key (order-preserving
    // integer keys, reset by the block that closes the step) and publishes
    // omega_span = max - min, so that omega_t[a] - omega_t[b] >= -omega_span for
    // any two cells of a type.  The move kernels use it to reject trials
    // without reading omega; +inf (after creation, scmf_set_omega or a
    // checkpoint read) disables that until the next field step.
    uint32_t om_max_key, om_min_key;
    float omega_span;
    uint32_t pad3;
    // the same in a launch of many sweeps (k_run): largest and smallest key of the
    // field step of each sweep, by its number mod 3
    uint32_t om_keys[3][2];
    unsigned long long slot_last[kSlots];  // k_run: accepted moves of its last sweep
    SweepSys sweep;
    BondConsts by_deg[kGraphDeg + 1];  // of a bead with that many bonds
    FieldSys field;
    // the statistics of the last sweep in the public layout, written by
    // k_stats_out for asynchronous reads (scmf_step_stats_async)
    scmf_stats stats_out;
};

// Work item of the move / grid kernel: a run of whole chains of one architecture.
struct MoveTile {
    SysDev* sys;
    const ArchDev* arch;
    int32_t chain0;       // first storage slot (system-wide chain index)
    int32_t n_chains;
    int64_t bead0;        // first bead (system arrays)
    int32_t n_tiles_sys;  // move tiles of this system in the launch
    int32_t arch_index;   // architecture of the tile within its system
};

// Work item of the move kernels of warp tiles: a run of whole chains of one architecture.
struct WarpTile {
    SysDev* sys;
    const ArchDev* arch;
    int64_t bead0;      // first bead (system arrays)
    uint32_t chain;     // first chain, counted in its architecture
    int32_t n_chains, n_beads, length;
};

// Work item of the field kernel: a run of cells of one system.
struct FieldTile {
    SysDev* sys;
    int64_t cell0;
    int32_t n_cells;
    int32_t n_tiles_sys;  // field tiles of this system in the launch
    int32_t first_tile;   // index of this system's first field tile in the launch
    int32_t pad;
};

// Bits of SysDev::error_word: a tile larger than k_sweep's shared memory; a warp's tile
// that did not arrive; blocks of a launch that did not come to a barrier.
constexpr uint32_t kErrorSize = 1u, kErrorTile = 4u, kErrorBarrier = 8u;
constexpr long long kWaitClocks = 4000000000ll;  // a wait in a kernel gives up after about two seconds
constexpr int kWaitShift = 10;

enum SweepMode : int { kMoveOnly = 0, kMoveGrid = 1, kGridOnly = 2 };

// What k_close does for each system of a launch.
enum CloseMode : int {
    kCloseMove = 1, kCloseField = 2, kCloseBond = 4, kCloseAdvance = 16,
    kCloseAverage = 32,  // count a time-averaged density sample when the sweep took one
    kSweepClose = kCloseMove | kCloseField | kCloseAdvance | kCloseAverage,
    kSweepOn = kSweepClose & ~kCloseField  // of a sweep that another one follows in the same call
};

// Per-tile partial sums of the chain observables (k_observables), each over
// the chains of one move tile, in double.
enum ObsSlot : int {
    kObsRe = 0,     // end-to-end vector components squared, x y z (first to last bead)
    kObsRg = 3,     // radius of gyration components squared
    kObsBond = 6,   // bond vector components squared, summed over bonds
    kObsMsd = 9,    // bead displacement from the reference snapshot, squared
    kObsMsdCom = 12,  // chain centre-of-mass displacement, squared
    kObsSlots = 16
};

// The tile ranges of one system in a launch's work lists.
struct SysClose {
    SysDev* sys;
    int32_t move_first, move_count;
    int32_t field_first, field_count;
};

// Launchers (scmf_kernels.cu).  Every pointer is device memory.
// fold_magic's offset and multiplier for an axis of n cells, 2 <= n <= 256.
inline int32_t fold_offset(uint32_t n) {
    const uint32_t bias = n * (((1u << 22) + n - 1) / n);  // a multiple of n, at least 2^22
    return (int32_t)(0x4B400000u - bias);
}
inline uint32_t fold_magic_of(uint32_t n) { return (uint32_t)(((1ull << 32) + n - 1) / n); }

// Round keys of Philox4x32-10 for one 64-bit key: round r XORs in
// (k0 + r * 0x9E3779B9, k1 + r * 0xBB67AE85) (mod 2^32).  Passed to a kernel
// by value, the schedule sits in the parameter constant bank, so each round's
// XOR reads its key there instead of advancing two key registers.
struct PhiloxKeys {
    uint32_t k[20];  // k[2r], k[2r + 1]: the two key words of round r
};

inline PhiloxKeys philox_schedule(uint32_t k0, uint32_t k1) {
    PhiloxKeys s;
    for (int r = 0; r < 10; ++r) {
        s.k[2 * r] = k0;
        s.k[2 * r + 1] = k1;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return s;
}

// The tiles of one architecture in a launch of one system: tile first + i has its
// chains i * per ... (i + 1) * per.
struct SweepArch {
    const ArchDev* arch;
    int64_t bead_base;
    int32_t first, per, n_chains, length;
};
constexpr int kSweepMaxArch = 4;

enum KeyMode { kKeysNone = 0, kKeysHigh = 1, kKeysBoth = 2 };

struct LaunchShape {
    int blocks;    // 0 = one CTA per tile
    int threads;
    int smem;      // unused by the launchers (they size shared memory themselves)
    int n_types;   // field kernel: monomer types shared by all systems, 0 = mixed
    // sweep kernel: kKeysBoth when every system of the launch has the seed of
    // `keys`, kKeysHigh when they share its upper 32 bits, else kKeysNone
    int keyed;
    PhiloxKeys keys;
    // every architecture of the launch fits a warp's tile (see tile_ranges)
    const WarpTile* warp_tiles;
    int n_warp_tiles;
    int form;           // SweepFormId
    int one;            // the launch has one system: `system`, with the constants `sweep` and n_arch tile ranges
    int once;           // the positions are more than L2 holds
    int chained;        // the kernel before in the stream is this plan's: the launch may begin beside its last blocks
    SysDev* system;
    SweepSys sweep;
    int n_arch;
    SweepArch arch[kSweepMaxArch];
};

// A system of a k_run launch and its field tiles.
struct RunSystem {
    SysDev* sys;
    int32_t field_first, field_count;
};

// What k_run needs besides SweepArgs.
struct RunArgs {
    const RunSystem* systems;
    const FieldTile* field;       // a warp's work each
    double* ef_part;              // field energy of every field tile after the last sweep
    unsigned long long* barrier;  // the grid barrier's count, and after it whether it is broken
    int n_sys, n_field, n_sweeps;
    uint32_t wait;                // how long a block waits for the others, in 2^kWaitShift clocks
};

// Parameters of the move kernels of warp tiles.
struct SweepArgs {
    const WarpTile* tiles;
    int n_tiles, move_counts, once, pad;
    PhiloxKeys keys;
    // one system
    SysDev* system;
    SweepSys sys;
    int n_arch;
    SweepArch arch[kSweepMaxArch];
};

// Forms of the move kernels of warp tiles: the warps of a CTA (one CTA per SM)
// and the beads of a warp's tile that shared memory then leaves room for.  Four
// warps a scheduler keep the screen's pipes busy, and longer tiles fill the warps
// of the resolve step better; half as many, with longer tiles still, where a chain
// is longer than that.  Systems that are not screened have a form without the
// screen's code, its table and the lists: 409,600 beads 13.1 us a sweep, 14.8 in
// the screened form (and 13.9, 15.8, 17.7 with 12, 28 and 24 warps of an SM, the
// last two short of registers).
// Plans with other bond graphs than linear chains have a form with the code for
// both, screened or not, and twelve warps: 2.0M beads in combs 25.1 us a sweep; with
// sixteen 28.5 (the screen of arbitrary neighbours does not fit 128 registers beside
// the exact trials), with eight 26.6.
// k_sweep_pairs has forms of its own, for one system of even chains and for any others:
// no buffers, as many warps as its registers leave, and tiles that only share out the work.
// 28 warps spill, 16 and 20 are too few (20.5M beads 222 us with 24 or 28, 245 with 20; in
// the second form 60 systems of 14M beads 308 us with 20, 352 with 16).
enum SweepFormId { kFormScreened = 0, kFormLong = 1, kFormUnscreened = 2, kFormGraph = 3, kFormPairs = 4, kFormPairsList = 5 };
struct SweepForm {
    int warps, beads;
};
constexpr SweepForm kSweepForms[6] = {{16, 960}, {8, 1984}, {16, 960}, {12, 1280}, {24, 1024}, {20, 1024}};
// Bead pairs of a tile of linear chains at most: a lane names the tile's pairs by the
// bits of a word, one for each row of 32.  A chain has half as many pairs as beads,
// rounded up: tiles of single beads, of trimers and of other short odd chains come to
// this before they come to the beads of a long form.
constexpr int kTilePairs = 32 * 32;
constexpr size_t kL2Bytes = 126u << 20;
// The screen of a system by x = A 4k: from which x it runs in plans with branched chains, in
// those of linear ones, and in these even where k_sweep_pairs could make every trial.  Below a line
// so many trials pass that making all of them is faster.  10M beads in chains of 33, x 2.4:
// screened 226 us a sweep, not 185; x 3.1: 137 and 174.  20.5M beads in chains of 32, x 3.1:
// screened 298, in k_sweep_pairs 216; x 3.7: 191 and 209.  10M beads in combs, x 1.96: 255 and
// 235; x 2.4: 210 and 229.
enum ScreenLevel : int { kScreenOff = 0, kScreenGraphs = 1, kScreenTiles = 2, kScreenAll = 3 };
constexpr float kScreenFromAc[4] = {0.0f, 2.0f, 2.8f, 3.4f};

// Streaming multiprocessors of the current device (read once per device; 148
// on a B200), for grid and tile sizing.
int sm_count();

int launch_init_coords(SysDev* d_sys, const ArchDev* d_arch, int n_arch, int n_chains, void* stream);
// Writes the statistics of the last sweep into d_sys->stats_out (one thread).
int launch_stats_out(SysDev* d_sys, void* stream);
// Copies the current counts (counts[cur], 32-bit words) into dst.
int launch_copy_counts(const SysDev* d_sys, uint32_t* dst, int64_t n_words, void* stream);
// Move kernels add their accept counts into SysDev::slot_acc (32-way spread);
// the field kernel writes one energy per tile into ef_part, the bond-energy
// kernel one per move tile into eb_part; k_close sums and publishes them.
int launch_sweep(int mode, const MoveTile* tiles, int n_tiles, int max_tile_beads, int max_length,
                 const LaunchShape& shape, void* stream);
// n_sweeps whole sweeps of a plan with warp tiles (shape.warp_tiles)
// in one cooperative launch.
int launch_run(const LaunchShape& shape, const RunArgs& run, void* stream);
// close_mode != 0: the last field tile of every system closes it in the same
// launch (what k_close does with that mode), so a sweep is two launches.
int launch_field(bool fused, int force_update, const FieldTile* tiles, int n_tiles, LaunchShape shape,
                 double* ef_part, int close_mode, void* stream);
int launch_bond_energy(const MoveTile* tiles, int n_tiles, LaunchShape shape, double* eb_part, void* stream);
// The systems' error words of a launch list, or'ed into *out.
int launch_error_words(const SysClose* list, int n_sys, uint32_t* out, void* stream);
int launch_close(const SysClose* list, int n_sys, const double* ef_part, const double* eb_part, int mode, void* stream);
int launch_aos_to_soa(const float* aos, SysDev* sys, const ArchDev* arch, int n_arch, int64_t n_beads,
                      void* stream);
// Storage beads [i0, i1) from AoS positions (storage order = chain order: the
// AoS bead of storage bead i is bead i), then their counts added into
// counts[0] (a cleared buffer): one chunk of a chunked coordinate upload.
int launch_aos_chunk(const float* aos, SysDev* sys, const ArchDev* arch, int n_arch, int64_t i0, int64_t i1,
                     void* stream);
int launch_soa_to_aos(float* aos, const SysDev* sys, const ArchDev* arch, int n_arch, int64_t n_beads,
                      void* stream);
int launch_unpack_counts16(const SysDev* sys, uint32_t* out, int64_t n, void* stream);
// Validation (scmf_validate): out[0] += non-finite positions, out[1] +=
// positions beyond the exact fold range; out[2] += differing count words of
// a and b, out[3] += non-finite omega; sums[t] += counts of type t.
int launch_validate_positions(const SysDev* sys, int64_t n_beads, unsigned long long* out, void* stream);
int launch_validate_cells(const SysDev* sys, const uint32_t* a, const uint32_t* b, int64_t n_words,
                          int64_t n_values, unsigned long long* out, unsigned long long* sums, void* stream);
// Adds the current counts into SysDev::avg and counts one sample.
int launch_average_sample(SysDev* sys, int64_t n, void* stream);
// Chain observables: kObsSlots partial sums per move tile into part; ref_xyz
// is the SoA reference snapshot (x, then y, then z; NULL = no displacements).
int launch_observables(const MoveTile* tiles, int n_tiles, const float* ref_xyz, int64_t n_beads_sys,
                       double* part, void* stream);
size_t sweep_smem_bytes(int max_tile_beads, int max_length);
// Field coefficients cf[t + n*s] in FP32 from xn[t + n*s] (double): diagonal
// xn/N_ref; off-diagonal -xn/(2 N_ref) (SCMF0) or xn/N_ref (literal).
void field_coefficients(int n, const double* xn, int nref, int hamiltonian, float* cf);
// Sets the thread's last-error message (scmf_engine.cpp); returns code.
scmf_status fail(scmf_status code, const char* fmt, ...);
int configure_kernels();
int launch_debug_math(uint32_t k0, uint32_t k1, int n, uint32_t* words, float* logs, float* normals, void* stream);

}  // namespace scmf
