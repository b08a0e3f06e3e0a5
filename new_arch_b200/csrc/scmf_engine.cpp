// Host engine of libscmf: specs, systems, work plans, the plain and batched
// step loops, and the C ABI entry points of include/scmf.h except file I/O
// (scmf_files.cpp) and serving (scmf_server.cpp).
//
// The reference's host orchestration (smc.cu:3-72, mesh.cu:161-248,
// mesh_mpi.cpp:4-27, test.cpp:37-43) launches one kernel at a time with a
// cudaDeviceSynchronize after each and a P2P/MPI density reduction.  Here a
// sweep is a share of one launch of many sweeps, two launches chained on one
// stream (fused move+grid, then field) or a replayed CUDA graph of these
// (DevPlan::run_sweeps), with no host round trip; the step counter, the counts
// and the statistics live on the device.
#include "scmf_engine.h"
#include "scmf_screen_table.h"

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <mutex>

namespace scmf {

static thread_local std::string g_last_error;

scmf_status fail(scmf_status code, const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_last_error = buf;
    return code;
}

void clear_error() { g_last_error.clear(); }
const char* last_error_cstr() { return g_last_error.c_str(); }

#define CK(expr)                                                                                   \
    do {                                                                                           \
        cudaError_t e_ = (expr);                                                                   \
        if (e_ != cudaSuccess) return fail(SCMF_E_CUDA, "%s: %s", #expr, cudaGetErrorString(e_)); \
    } while (0)

#define CKL(expr)                                                                                      \
    do {                                                                                               \
        int e_ = (expr);                                                                               \
        if (e_ != 0)                                                                                   \
            return fail(SCMF_E_CUDA, "%s: %s", #expr, cudaGetErrorString((cudaError_t)e_));          \
    } while (0)

scmf_status dev_alloc(void** p, size_t bytes, cudaStream_t st) {
    static std::once_flag once;
    std::call_once(once, [] {
        int dev = 0;
        cudaMemPool_t pool;
        if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
            uint64_t keep = UINT64_MAX;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        }
        cudaGetLastError();
    });
    bytes = (std::max<size_t>(bytes, 16) + 255) / 256 * 256;
    cudaError_t e = cudaMallocAsync(p, bytes, st);
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return fail(e == cudaErrorMemoryAllocation ? SCMF_E_NOMEM : SCMF_E_CUDA, "cudaMallocAsync(%zu): %s", bytes,
                    cudaGetErrorString(e));
    }
    return SCMF_OK;
}

void dev_free(void* p, cudaStream_t st) {
    if (p) cudaFreeAsync(p, st);
}

// ceil(2^32 / n): for i * n < 2^32, i / n == umulhi(i, magic).  n == 1 has no
// 32-bit magic; the kernels test for it.
uint32_t magic_for(uint32_t n) {
    if (n <= 1) return 0u;
    return (uint32_t)((((uint64_t)1 << 32) + n - 1) / n);
}

scmf_status validate_spec(const scmf_spec& s) {
    if (s.n_types < 1 || s.n_types > kMaxTypes) return fail(SCMF_E_INVALID, "n_mono_types %d not in [1,%d]", s.n_types, kMaxTypes);
    if (s.nx < 1 || s.ny < 1 || s.nz < 1) return fail(SCMF_E_INVALID, "grid %d x %d x %d invalid", s.nx, s.ny, s.nz);
    if ((int64_t)s.nx * s.ny * s.nz > ((int64_t)1 << 30)) return fail(SCMF_E_INVALID, "grid too large");
    // the FP32 cell fold is exact while |x / dx| < 2^22: keep whole boxes well inside that
    if (s.nx > (1 << 20) || s.ny > (1 << 20) || s.nz > (1 << 20))
        return fail(SCMF_E_INVALID, "grid axis longer than %d cells", 1 << 20);
    if (!(s.lx > 0 && s.ly > 0 && s.lz > 0)) return fail(SCMF_E_INVALID, "box lengths must be positive");
    if ((int)s.xn.size() != s.n_types * s.n_types) return fail(SCMF_E_INVALID, "xn matrix not set");
    if (s.p.reference_nbeads < 1) return fail(SCMF_E_INVALID, "reference_nbeads must be >= 1");
    if (!(s.p.smc_a >= 0) || !std::isfinite(s.p.harmonic_normb)) return fail(SCMF_E_INVALID, "bad smc_a / harmonic_normb");
    if (s.p.count_bits != 16 && s.p.count_bits != 32) return fail(SCMF_E_INVALID, "count_bits must be 16 or 32");
    if (s.p.hamiltonian != SCMF_HAM_SCMF0 && s.p.hamiltonian != SCMF_HAM_LITERAL) return fail(SCMF_E_INVALID, "unknown hamiltonian");
    if (s.p.field_rule != SCMF_FIELD_REFERENCE && s.p.field_rule != SCMF_FIELD_EVERY) return fail(SCMF_E_INVALID, "unknown field rule");
    if (s.archs.empty()) return fail(SCMF_E_INVALID, "spec has no polymer architecture");
    int64_t beads = 0, chains = 0;
    for (const auto& a : s.archs) {
        if (a.length < 1 || a.length > kMaxLength) return fail(SCMF_E_INVALID, "chain length %d not in [1,%d]", a.length, kMaxLength);
        if (a.n_chains < 0) return fail(SCMF_E_INVALID, "negative chain count %d", a.n_chains);
        beads += (int64_t)a.length * a.n_chains;
        chains += a.n_chains;
    }
    if (beads <= 0) return fail(SCMF_E_INVALID, "system has no beads");
    if (beads >= ((int64_t)1 << 31) || chains >= ((int64_t)1 << 31)) return fail(SCMF_E_INVALID, "too many beads");
    if (s.p.count_bits == 16 && beads >= 65536)
        return fail(SCMF_E_INVALID, "16-bit counts need fewer than 65536 beads (%lld)", (long long)beads);
    return SCMF_OK;
}

scmf_status prepare_archs(const scmf_spec& s, std::vector<ArchHost>* out, int64_t* n_beads, int* n_chains) {
    out->clear();
    int64_t nb = 0;
    int nc = 0;
    for (const auto& a : s.archs) {
        ArchHost h;
        h.length = a.length;
        h.n_chains = a.n_chains;
        h.chain_base = nc;
        h.bead_base = nb;
        h.init_sigma = (float)(a.init_sigma > 0 ? a.init_sigma : (a.length > 1 ? 1.0 / std::sqrt(3.0 * (a.length - 1.0)) : 0.0));
        const int L = a.length;
        h.beads.assign(L, BeadInfo{});
        std::vector<std::vector<char>> adj(L, std::vector<char>(L, 0));
        for (size_t b = 0; b + 1 < a.bonds.size(); b += 2) {
            int i = a.bonds[b], j = a.bonds[b + 1];
            if (i < 0 || j < 0 || i >= L || j >= L || i == j) return fail(SCMF_E_INVALID, "bond (%d,%d) out of range", i, j);
            adj[i][j] = adj[j][i] = 1;
        }
        for (int i = 0; i < L; ++i) {
            if (a.type[i] < 0 || a.type[i] >= s.n_types) return fail(SCMF_E_INVALID, "monomer type %d out of range", a.type[i]);
            BeadInfo& bi = h.beads[i];
            bi.type = (uint8_t)a.type[i];
            int d = 0;
            for (int j = 0; j < L; ++j)
                if (adj[i][j]) {
                    if (d >= kMaxDeg) return fail(SCMF_E_INVALID, "bead %d has more than %d bonds", i, kMaxDeg);
                    bi.nbr[d++] = (uint16_t)j;
                }
            bi.deg = (uint8_t)d;
            h.max_deg = std::max(h.max_deg, d);
        }
        // greedy colouring in index order
        int ncol = 0;
        for (int i = 0; i < L; ++i) {
            unsigned used = 0;
            for (int d = 0; d < h.beads[i].deg; ++d) {
                int j = h.beads[i].nbr[d];
                if (j < i) used |= 1u << h.beads[j].color;
            }
            int c = 0;
            while (used & (1u << c)) ++c;
            if (c >= kMaxColors) return fail(SCMF_E_INVALID, "architecture needs more than %d colours", kMaxColors);
            h.beads[i].color = (uint8_t)c;
            ncol = std::max(ncol, c + 1);
        }
        h.n_colors = ncol;
        h.linear = true;
        for (int i = 0; i < L && h.linear; ++i) {
            const BeadInfo& bi = h.beads[i];
            const int want = (i > 0) + (i + 1 < L);
            if (bi.deg != want || bi.color != (i & 1)) h.linear = false;
            if (bi.deg >= 1 && i > 0 && bi.nbr[0] != i - 1) h.linear = false;
            if (i + 1 < L && bi.nbr[bi.deg - 1] != i + 1) h.linear = false;
        }
        h.color_beads.clear();
        for (int c = 0; c < ncol; ++c) {
            h.color_off[c] = (int)h.color_beads.size();
            for (int i = 0; i < L; ++i)
                if (h.beads[i].color == c) h.color_beads.push_back((uint16_t)i);
        }
        h.color_off[ncol] = (int)h.color_beads.size();
        nb += (int64_t)L * a.n_chains;
        nc += a.n_chains;
        out->push_back(std::move(h));
    }
    *n_beads = nb;
    *n_chains = nc;
    return SCMF_OK;
}

static size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

static size_t count_words(const scmf_spec& s) {
    const size_t cells = (size_t)s.nx * s.ny * s.nz * s.n_types;
    return s.p.count_bits == 16 ? (cells + 1) / 2 : cells;
}

size_t system_device_bytes(const scmf_spec& s) {
    int64_t beads = 0, chains = 0, arch_bytes = 0;
    for (const auto& a : s.archs) {
        beads += (int64_t)a.length * a.n_chains;
        chains += a.n_chains;
        arch_bytes += round_up((size_t)a.length * (sizeof(BeadInfo) + 3 + sizeof(GraphBead)) + 16, 256);
    }
    const size_t cells = (size_t)s.nx * s.ny * s.nz * s.n_types;
    size_t b = 3 * round_up((size_t)(beads + 4) * 4, 256) + round_up((size_t)chains * 4, 256);
    b += 2 * round_up(count_words(s) * 4, 256) + round_up(cells * 4, 256);
    b += round_up(sizeof(SysDev), 256) + round_up(s.archs.size() * sizeof(ArchDev), 256) + arch_bytes;
    b += (size_t)chains / 8 * sizeof(MoveTile) + 64 * 1024;  // work lists
    return b;
}

void field_coefficients(int n, const double* xn, int nref, int hamiltonian, float* cf) {
    const double inv_n = 1.0 / (double)nref;
    for (int i = 0; i < kMaxTypes * kMaxTypes; ++i) cf[i] = 0.0f;
    for (int t = 0; t < n; ++t)
        for (int u = 0; u < n; ++u) {
            const double v = xn[t + n * u];
            float c;
            if (t == u) c = (float)(v * inv_n);
            else if (hamiltonian == SCMF_HAM_SCMF0) c = (float)(-0.5 * v * inv_n);
            else c = (float)(v * inv_n);
            cf[t + n * u] = c;
        }
}

// Constants of the move kernel's screen (ScreenDev), rounded towards passing a
// trial.  Off where they leave the range in which the bounds there hold, and
// where proposals are small enough that most trials would pass: with x = A 4k,
// 4k the c of an inner bead, |v|^2 has (x^2 + 1) / (2 x) times the mean of the
// limit's |f|^2 term, so screened trials pass often below x of about 2.
constexpr double kScreenEta = 0x1p-6, kScreenUnit = 0x1p30;
static float rounded_up(double v) { return std::nextafterf((float)v, INFINITY); }

// a and b for beads of g bonds; false where they are out of range.
static bool screen_of(const SysDev& d, int g, float* a, float* b) {
    const double K = (1.0 + kScreenEta) * (1.0 + 0x1p-10), A = d.A, R = d.R, c = d.cdeg[g];
    const double bg = K / (c * c * R * R);
    *a = (float)((A - 1.0 / c) / R * kScreenUnit);
    *b = rounded_up(bg * kScreenUnit * kScreenUnit);
    for (const double v : {A, R, c, (double)d.ac4deg[g], bg})
        if (!(v > 1e-12 && v < 1e12)) return false;
    return true;
}

static ScreenDev screen_constants(const SysDev& d) {
    ScreenDev s{};
    const double delta = SCMF_SCREEN_DELTA, A = d.A;
    for (int level = kScreenGraphs; level <= kScreenAll; ++level)
        if (A > 0.0 && A * (double)d.cdeg[2] >= kScreenFromAc[level]) s.on = level;
    s.add = rounded_up((1.0 + 1.0 / kScreenEta) * 3.0 * delta * delta * kScreenUnit * kScreenUnit);
    s.u = rounded_up(4.0 / A);
    for (int g = 1; g <= 2; ++g)
        if (!screen_of(d, g, &s.a[g], &s.b[g])) s.on = kScreenOff;
    return s;
}

void fill_sysdev_constants(const scmf_spec& s, int64_t n_beads, SysDev* d) {
    d->stop_step = 0xFFFFFFFFu;
    d->om_max_key = 0u;            // identities of the running max / min
    d->om_min_key = 0xFFFFFFFFu;
    d->omega_span = INFINITY;      // no bound until a field step computes one
    d->n_types = s.n_types;
    d->nx = s.nx; d->ny = s.ny; d->nz = s.nz;
    d->n_cells = (int64_t)s.nx * s.ny * s.nz;
    d->n_beads = n_beads;
    // derived constants (init_config.cu:480-484, 565-567, 785, 807-808) rounded to FP32
    d->inv_dx = (float)((double)s.nx / s.lx);
    d->inv_dy = (float)((double)s.ny / s.ly);
    d->inv_dz = (float)((double)s.nz / s.lz);
    d->lx = (float)s.lx; d->ly = (float)s.ly; d->lz = (float)s.lz;
    d->scale = (float)((double)d->n_cells / (double)n_beads);
    d->k = (float)s.p.harmonic_normb;
    d->k2 = (float)(2.0 * s.p.harmonic_normb);
    d->A = (float)s.p.smc_a;
    d->R = (float)std::sqrt(2.0 * s.p.smc_a);
    for (int g = 0; g <= kMaxDeg; ++g) {
        d->cdeg[g] = d->k2 * (float)g;
        d->ac4deg[g] = (d->A * d->cdeg[g]) * 0.25f;
    }
    field_coefficients(s.n_types, s.xn.data(), s.p.reference_nbeads, s.p.hamiltonian, d->cf);
    d->hamiltonian = s.p.hamiltonian;
    d->field_rule = s.p.field_rule;
    d->count16 = s.p.count_bits == 16 ? 1 : 0;
    d->n_arch = (int)s.archs.size();
    d->seed_lo = (uint32_t)s.p.seed;
    d->seed_hi = (uint32_t)(s.p.seed >> 32);
}

void fill_sweep_constants(SysDev* d) {
    SweepSys& w = d->sweep;
    w.x = d->x;
    w.y = d->y;
    w.z = d->z;
    w.omega = d->omega;
    w.counts = d->counts[0];
    w.n_cells = (uint32_t)d->n_cells;
    w.k2 = d->k2;
    w.A = d->A;
    w.R = d->R;
    const float inv[3] = {d->inv_dx, d->inv_dy, d->inv_dz};
    const int n[3] = {d->nx, d->ny, d->nz};
    bool pow2 = true, small = true;
    for (int i = 0; i < 3; ++i) {
        w.inv_d[i] = inv[i];
        w.n[i] = n[i];
        pow2 = pow2 && (n[i] & (n[i] - 1)) == 0;
        small = small && n[i] >= 2 && n[i] <= 256;
    }
    w.fold = pow2 ? 0 : small ? 1 : 2;
    for (int i = 0; i < 3 && w.fold == 1; ++i) {
        w.fold_off[i] = fold_offset((uint32_t)n[i]);
        w.fold_mag[i] = fold_magic_of((uint32_t)n[i]);
    }
    for (int g = 0; g < 3; ++g) {
        w.cdeg[g] = d->cdeg[g];
        w.ac4[g] = d->ac4deg[g];
    }
    w.seed_lo = d->seed_lo;
    w.seed_hi = d->seed_hi;
    w.count16 = d->count16;
    w.screen = screen_constants(*d);
    d->by_deg[0] = BondConsts{0.0f, INFINITY, 0.0f, 0.0f};  // no bond, nothing to screen by
    for (int g = 1; g <= kGraphDeg; ++g) {
        float a, b;
        if (!screen_of(*d, g, &a, &b)) w.screen.on = kScreenOff;
        d->by_deg[g] = BondConsts{a, b, d->cdeg[g], d->ac4deg[g]};
    }
    FieldSys& f = d->field;
    f.counts = d->counts[0];
    f.omega = d->omega;
    f.n_cells = d->n_cells;
    f.scale = d->scale;
    f.n_types = d->n_types;
    f.literal = d->hamiltonian == SCMF_HAM_LITERAL ? 1 : 0;
    f.count16 = d->count16;
    f.rule = d->field_rule;
    for (int i = 0; i < kMaxTypes * kMaxTypes; ++i) f.cf[i] = d->cf[i];
}

scmf_tune default_tune() {
    scmf_tune t{};
    t.chains_per_tile = 0;
    t.threads_move = 128;  // 4 warps: CTAs retire and refill at a finer grain than 8-warp CTAs
    t.cells_per_tile = 0;
    t.threads_field = 256;
    t.persistent_ctas = 0;
    t.use_graph = 1;
    return t;
}

scmf_tune resolve_tune(const scmf_tune* t) {
    scmf_tune r = default_tune();
    if (!t) return r;
    if (t->chains_per_tile > 0) r.chains_per_tile = t->chains_per_tile;
    if (t->threads_move > 0) r.threads_move = std::min(256, std::max(32, t->threads_move / 32 * 32));
    if (t->cells_per_tile > 0) r.cells_per_tile = t->cells_per_tile;
    if (t->threads_field > 0) r.threads_field = std::min(256, std::max(32, t->threads_field / 32 * 32));
    r.persistent_ctas = std::max(0, t->persistent_ctas);
    r.use_graph = t->use_graph;
    r.beads_per_tile = std::max(0, std::min(t->beads_per_tile, kMaxTileBeads));
    return r;
}


void DevPlan::release() {
    if (graph) cudaGraphExecDestroy(graph);
    if (graph_src) cudaGraphDestroy(graph_src);
    void* ptrs[] = {d_move, d_field, d_close, tiles.list, single.list == tiles.list ? nullptr : single.list, d_ef, d_eb, d_run};
    for (void* p : ptrs) dev_free(p, stream);
    graph = nullptr;
    graph_src = nullptr;
    d_move = nullptr;
    d_field = nullptr;
    d_close = nullptr;
    tiles = single = WarpTiles{};
    d_run = nullptr;
    d_ef = nullptr;
    d_eb = nullptr;
    n_move = n_field = n_sys = n_warp = 0;
}

// The tiles of the move kernels of warp tiles: whole chains of one architecture, as many chains in
// each (SweepArch::per).  Every warp of the GPU gets the same number of tiles, of
// sizes up to what its buffer holds and no smaller than a row of 32 bead pairs.
// A tile of linear chains also has no more than kTilePairs bead pairs.  Empty for a plan
// that the kernel does not take.
static std::vector<SweepArch> form_ranges(const Plan& p, int form) {
    std::vector<SweepArch> out;
    const int cap = kSweepForms[form].beads;
    const int64_t warps = (int64_t)sm_count() * kSweepForms[form].warps;
    int64_t beads = 0;
    const auto chains_at_most = [&](const Plan::Chains& c) {
        return c.linear ? std::min(cap / c.length, kTilePairs / ((c.length + 1) / 2)) : cap / c.length;
    };
    int most = cap;  // what a tile of every architecture can reach
    for (const auto& c : p.chains) {
        beads += (int64_t)c.length * c.n_chains;
        most = std::min(most, chains_at_most(c) * c.length);
    }
    const int64_t turns = std::max<int64_t>(1, (beads + warps * most - 1) / (warps * most));  // tiles of a warp
    const auto per_tile = [&](const Plan::Chains& c, int64_t target) {
        return (int)std::min<int64_t>(chains_at_most(c), std::max<int64_t>(1, (target + c.length - 1) / c.length));
    };
    int64_t target = std::max<int64_t>(64, (beads + warps * turns - 1) / (warps * turns));
    for (; target < cap; target += std::max<int64_t>(1, target / 64)) {  // the last tile of each architecture is a part
        int64_t n = 0;
        for (const auto& c : p.chains) n += (c.n_chains + per_tile(c, target) - 1) / per_tile(c, target);
        if (n <= warps * turns) break;
    }
    int first = 0;
    for (const auto& c : p.chains) {
        SweepArch r{c.arch, c.bead_base, first, per_tile(c, target), c.n_chains, c.length};
        first += (c.n_chains + r.per - 1) / r.per;
        out.push_back(r);
    }
    return out;
}

static int tiles_of(const std::vector<SweepArch>& ranges) {
    return ranges.empty() ? 0 : ranges.back().first + (ranges.back().n_chains + ranges.back().per - 1) / ranges.back().per;
}

// The tiles of k_sweep_pairs, where at least three lanes of four have a pair; empty otherwise.
static std::vector<SweepArch> pairs_ranges(const Plan& p, int* form) {
    int64_t pairs = 0, lanes = 0;
    bool even = p.cells.size() == 1 && p.chains.size() <= kSweepMaxArch;
    for (const auto& c : p.chains) {
        if (!c.linear || c.length > 64) return {};
        const int h = (c.length + 1) / 2, per = 32 / h;
        pairs += (int64_t)h * c.n_chains;
        lanes += (int64_t)32 * ((c.n_chains + per - 1) / per);
        even = even && (c.length | c.bead_base) % 2 == 0;
    }
    if (4 * pairs < 3 * lanes) return {};
    *form = even ? kFormPairs : kFormPairsList;
    return form_ranges(p, *form);
}

std::vector<SweepArch> tile_ranges(const Plan& p, int* form) {
    if (p.chains.empty() || !p.cells32 || p.max_deg > kGraphDeg) return {};
    int64_t beads = 0, exact = 0;  // all, and those of chains whose trials k_sweep_pairs makes as fast as a screen does
    bool screened = false;
    for (const auto& c : p.chains) {
        beads += (int64_t)c.length * c.n_chains;
        exact += c.screen < kScreenAll ? (int64_t)c.length * c.n_chains : 0;
        screened = screened || c.screen >= kScreenTiles;
    }
    *form = !p.linear ? kFormGraph : screened ? kFormScreened : kFormUnscreened;
    if (p.linear && p.max_length > kSweepForms[*form].beads) *form = kFormLong;
    if (p.max_length > kSweepForms[*form].beads) return {};
    std::vector<SweepArch> out = form_ranges(p, *form);
    // Trials that are all made exactly are made faster in registers (k_sweep_pairs) than in tiles, from 352 beads a warp
    // on also than in k_run: a sweep of 0.4M beads 12.4 us in k_run and 16.0 so, 0.8M 21.3 and 18.9 (in chains of 48 or 64
    // 19.4 and 20.3, 19.0 and 19.7), 2.0M 46.1 and 33.5, 20.5M 379 (in tiles) and 223.  So are those of many systems of
    // which a quarter of the beads is not screened: 32M beads, 25 % 467 us in tiles and 432 so, 50 % 634 and 452, 10 % 350 and
    // 399.
    const int64_t warps = (int64_t)sm_count() * kSweepForms[*form].warps;
    if (exact == beads ? beads > 352 * warps : tiles_of(out) > warps && 4 * exact >= beads) {
        std::vector<SweepArch> in_pairs = pairs_ranges(p, form);
        if (!in_pairs.empty()) return in_pairs;
    }
    return out;
}

static std::vector<WarpTile> tile_list(const Plan& p, const std::vector<SweepArch>& ranges) {
    std::vector<WarpTile> out;
    out.reserve((size_t)tiles_of(ranges));
    for (size_t k = 0; k < ranges.size(); ++k) {
        const SweepArch& r = ranges[k];
        for (int i = 0; i < r.n_chains; i += r.per) {
            const int n = std::min(r.per, r.n_chains - i);
            out.push_back({p.chains[k].sys, r.arch, r.bead_base + (int64_t)i * r.length, (uint32_t)i, n, n * r.length, r.length});
        }
    }
    return out;
}

// The warps of a launch of n_warp tiles that are made at once.
static int launched_warps(int n_warp, int form) {
    const int grid = std::min(n_warp, sm_count());
    return grid * std::min(kSweepForms[form].warps, (n_warp + grid - 1) / grid);
}

// Whether a plan's sweeps go many to a launch (k_run): a tile a warp, and no more cells
// than these warps can make omega of in the time that the launches of two kernels take.
// A step of a warp over its cells takes 0.6 us where few warps run, so up to 12 steps are
// as fast as k_field's launch over the whole GPU, and up to 27 where most of the GPU's
// warps run.  A sweep in one launch against two: 300 chains of 32 on 64^3 cells (7 steps)
// 10.8 and 12.0 us, on 80^3 (14) 14.8 and 12.7, on 128^3 (55) 40.8 and 16.0; 40 chains on
// 64^3 (102) 67 and 12; 1,000 on 96^3 (12) 14.0 and 14.0; 60,000 on 200^3 (26) 55.8 and
// 58.5; 10,000 on 256^3 (55) 90.7 and 77.2; 1,000 with four types on 96^3 (47) 98.6 and 39.4.
static bool runs_at_once(const Plan& p, int n_warp, int form) {
    const int all = sm_count() * kSweepForms[form].warps;
    if (n_warp < 1 || n_warp > all || form == kFormPairs || form == kFormPairsList) return false;
    const int warps = launched_warps(n_warp, form);
    int64_t cells = 0;
    for (const auto& c : p.cells) cells += c.second;
    return cells <= (int64_t)warps * (p.cells4 ? 128 : 32) * (4 * (int64_t)warps >= 3 * (int64_t)all ? 27 : 12);
}

// The tables of k_run as one buffer, its pointers still offsets: field tiles of a
// warp each, so that the warps of the launch share the cells evenly.
static std::vector<char> run_tables(const Plan& p, int n_warp, int form, RunArgs* run) {
    const int warps = launched_warps(n_warp, form);
    int64_t cells = 0;
    for (const auto& c : p.cells) cells += c.second;
    // whole rows of four cells a lane, or of one where that leaves warps idle
    const int64_t row = cells >= 128 * (int64_t)warps ? 128 : 32;
    const int64_t per = ((cells + warps - 1) / warps + row - 1) / row * row;
    std::vector<RunSystem> systems;
    std::vector<FieldTile> field;
    for (const auto& c : p.cells) {
        RunSystem rs{c.first, (int32_t)field.size(), 0};
        for (int64_t i = 0; i < c.second; i += per) {
            FieldTile t{};
            t.sys = c.first;
            t.cell0 = i;
            t.n_cells = (int32_t)std::min(per, c.second - i);
            field.push_back(t);
        }
        rs.field_count = (int32_t)field.size() - rs.field_first;
        systems.push_back(rs);
    }
    const size_t at_field = round_up(64 + systems.size() * sizeof(RunSystem), 64);
    const size_t at_ef = round_up(at_field + field.size() * sizeof(FieldTile), 64);
    std::vector<char> image(at_ef + field.size() * sizeof(double), 0);  // the barrier's count first
    std::memcpy(image.data() + 64, systems.data(), systems.size() * sizeof(RunSystem));
    std::memcpy(image.data() + at_field, field.data(), field.size() * sizeof(FieldTile));
    *run = RunArgs{};
    run->barrier = nullptr;
    run->wait = (uint32_t)(kWaitClocks >> kWaitShift);
    run->systems = (const RunSystem*)(size_t)64;
    run->field = (const FieldTile*)at_field;
    run->ef_part = (double*)at_ef;
    run->n_sys = (int)systems.size();
    run->n_field = (int)field.size();
    return image;
}

scmf_status DevPlan::upload(const Plan& p, const scmf_tune& t, cudaStream_t st) {
    release();
    stream = st;
    tune = t;
    n_move = (int)p.move.size();
    n_field = (int)p.field.size();
    max_tile_beads = p.max_tile_beads;
    max_length = p.max_length;
    n_types_uniform = p.n_types_uniform;
    one_seed = p.one_seed && !p.close.empty();
    one_seed_hi = p.one_seed_hi && !p.close.empty();
    seed = p.seed;
    n_sys = (int)p.close.size();
    system = n_sys == 1 ? p.close[0].sys : nullptr;
    std::vector<WarpTile> lists[2];
    const auto place = [&](const std::vector<SweepArch>& ranges, int form, WarpTiles* w, std::vector<WarpTile>* list) -> scmf_status {
        w->form = form;
        w->n = tiles_of(ranges);
        w->one = n_sys == 1 && ranges.size() <= kSweepMaxArch && form != kFormPairsList;
        if (w->one) {
            w->n_arch = (int)ranges.size();
            std::copy(ranges.begin(), ranges.end(), w->arch);
            return SCMF_OK;
        }
        *list = tile_list(p, ranges);
        scmf_status e = dev_alloc((void**)&w->list, std::max<size_t>(1, list->size()) * sizeof(WarpTile), st);
        if (!e && !list->empty())
            CK(cudaMemcpyAsync(w->list, list->data(), list->size() * sizeof(WarpTile), cudaMemcpyHostToDevice, st));
        return e;
    };
    int form = kFormScreened;
    const std::vector<SweepArch> ranges = tile_ranges(p, &form);
    scmf_status rc = place(ranges, form, &tiles, &lists[0]);
    if (rc) return rc;
    // A launch of one sweep has none of what makes k_run the faster of the two for few unscreened beads: 0.4M beads 18.9 us
    // a sweep in tiles and 16.1 in pairs, 0.8M 25.5 and 19.4, 10,000 11.2 and 10.4.
    single = tiles;
    if (form == kFormUnscreened) {
        const std::vector<SweepArch> in_pairs = pairs_ranges(p, &form);
        if (!in_pairs.empty()) {
            single = WarpTiles{};
            if ((rc = place(in_pairs, form, &single, &lists[1]))) return rc;
        }
    }
    n_warp = single.n;
    sweep = p.sweep;
    once = p.position_bytes > kL2Bytes / 2;
    const size_t nm = std::max<size_t>(1, p.move.size()), nf = std::max<size_t>(1, p.field.size());
    if ((rc = dev_alloc((void**)&d_move, nm * sizeof(MoveTile), st)) ||
        (rc = dev_alloc((void**)&d_field, nf * sizeof(FieldTile), st)) ||
        (rc = dev_alloc((void**)&d_close, (p.close.size() + 1) * sizeof(SysClose), st)) ||  // and the word of check()
        (rc = dev_alloc((void**)&d_ef, nf * sizeof(double), st)) || (rc = dev_alloc((void**)&d_eb, nm * sizeof(double), st)))
        return rc;
    CK(cudaMemcpyAsync(d_move, p.move.data(), p.move.size() * sizeof(MoveTile), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(d_field, p.field.data(), p.field.size() * sizeof(FieldTile), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(d_close, p.close.data(), p.close.size() * sizeof(SysClose), cudaMemcpyHostToDevice, st));
    std::vector<char> run_image;
    if (runs_at_once(p, tiles.n, tiles.form)) {
        run_image = run_tables(p, tiles.n, tiles.form, &run);
        if ((rc = dev_alloc(&d_run, run_image.size(), st))) return rc;
        CK(cudaMemcpyAsync(d_run, run_image.data(), run_image.size(), cudaMemcpyHostToDevice, st));
        const auto at = [&](const void* offset) { return (char*)d_run + (size_t)offset; };
        run.systems = (const RunSystem*)at(run.systems);
        run.field = (const FieldTile*)at(run.field);
        run.ef_part = (double*)at(run.ef_part);
        run.barrier = (unsigned long long*)at(run.barrier);
    }
    // the host vectors may go away after return: wait for the (pageable) copies
    CK(cudaStreamSynchronize(st));
    return SCMF_OK;
}

LaunchShape DevPlan::move_shape(bool many) const {
    const WarpTiles& w = many ? tiles : single;
    LaunchShape sh{};
    sh.blocks = tune.persistent_ctas > 0 ? std::min(tune.persistent_ctas, n_move) : 0;
    sh.threads = tune.threads_move;
    sh.n_types = n_types_uniform;
    sh.keyed = one_seed ? kKeysBoth : (one_seed_hi ? kKeysHigh : kKeysNone);
    sh.keys = philox_schedule((uint32_t)seed, (uint32_t)(seed >> 32));
    sh.warp_tiles = w.list;
    sh.n_warp_tiles = w.n;
    sh.form = w.form;
    sh.one = w.one ? 1 : 0;
    sh.system = system;
    sh.n_arch = w.n_arch;
    for (int i = 0; i < sh.n_arch; ++i) sh.arch[i] = w.arch[i];
    sh.once = once ? 1 : 0;
    sh.sweep = sweep;
    return sh;
}

LaunchShape DevPlan::field_shape() const {
    LaunchShape sh{};
    sh.blocks = tune.persistent_ctas > 0 ? std::min(tune.persistent_ctas, n_field) : 0;
    sh.threads = tune.threads_field;
    sh.n_types = n_types_uniform;
    return sh;
}

scmf_status DevPlan::enqueue_close(int mode, cudaStream_t st) const {
    CKL(launch_close(d_close, n_sys, d_ef, d_eb, mode, st));
    return SCMF_OK;
}

scmf_status DevPlan::check(cudaStream_t st) const {
    uint32_t any = 0, *const d_any = reinterpret_cast<uint32_t*>(d_close + n_sys);
    CKL(launch_error_words(d_close, n_sys, d_any, st));
    CK(cudaMemcpyAsync(&any, d_any, sizeof any, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (any) return fail(SCMF_E_DEVICE, "kernel error word 0x%x", any);
    return SCMF_OK;
}

scmf_status DevPlan::enqueue_sweep(cudaStream_t st, bool last) const {
    LaunchShape move = move_shape(), field = field_shape();
    move.chained = field.chained = n_warp > 0 ? 1 : 0;
    CKL(launch_sweep(kMoveGrid, d_move, n_move, max_tile_beads, max_length, move, st));
    CKL(launch_field(true, 0, d_field, n_field, field, d_ef, last ? kSweepClose : kSweepOn, st));
    return SCMF_OK;
}

scmf_status DevPlan::enqueue_move(cudaStream_t st) const {
    CKL(launch_sweep(kMoveGrid, d_move, n_move, max_tile_beads, max_length, move_shape(), st));
    return SCMF_OK;
}

scmf_status DevPlan::enqueue_field(cudaStream_t st) const {
    CKL(launch_field(true, 0, d_field, n_field, field_shape(), d_ef, kSweepClose, st));
    return SCMF_OK;
}

scmf_status DevPlan::run_sweeps(cudaStream_t st, int n) {
    if (n <= 0) return SCMF_OK;
    // A single sweep is two launches, of which the second begins beside the first: a cooperative launch, its barriers
    // and the positions' way back cost more than they save (enqueued one by one: 32,000 beads 13.4 us against 17.4,
    // 2.0M beads 22.4 against 32.8; two sweeps a call are the same either way, three faster in one launch).
    if (d_run && n > 1) {
        // some milliseconds a launch, so that other work on the GPU gets its turn
        const LaunchShape sh = move_shape(true);
        for (RunArgs r = run; n > 0; n -= r.n_sweeps) {
            r.n_sweeps = std::min(n, 1024);
            const int e = launch_run(sh, r, st);
            if (e == (int)cudaErrorCooperativeLaunchTooLarge) {  // a context that has not all of the GPU's SMs
                cudaGetLastError();
                break;
            }
            CKL(e);
        }
        if (n <= 0) return SCMF_OK;
    }
    // A sweep of warp tiles that do not all fit on the chip takes 50 us and more, so launching its two kernels one by one
    // keeps ahead of the GPU, and each may begin (tables, descriptors) beside the last blocks of the one before, which
    // replaying a graph of one sweep does not give: 4.7M beads in 20 systems 53.3 -> 49.3 us, 51.2M beads 336 -> 328.
    if (tune.use_graph && n_warp == 0) {
        if (!graph) {
            CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
            scmf_status rc = enqueue_sweep(st, true);
            cudaGraph_t g = nullptr;
            cudaError_t e = cudaStreamEndCapture(st, &g);
            if (rc != SCMF_OK) {
                if (g) cudaGraphDestroy(g);
                return rc;
            }
            if (e != cudaSuccess) return fail(SCMF_E_CUDA, "graph capture: %s", cudaGetErrorString(e));
            graph_src = g;
            CK(cudaGraphInstantiate(&graph, g, 0));
        }
        for (int i = 0; i < n; ++i) CK(cudaGraphLaunch(graph, st));
        return SCMF_OK;
    }
    for (int i = 0; i < n; ++i) {
        scmf_status rc = enqueue_sweep(st, i + 1 == n);
        if (rc) return rc;
    }
    return SCMF_OK;
}

scmf_status fetch_sysdev(const scmf_system* s, SysDev* out) {
    CK(cudaMemcpyAsync(out, s->d_sys, sizeof(SysDev), cudaMemcpyDeviceToHost, s->stream));
    CK(cudaStreamSynchronize(s->stream));
    return SCMF_OK;
}

}  // namespace scmf

using namespace scmf;

// Work tiles of this system appended to a plan.
scmf_status scmf_system::append_plan(const scmf_tune& t, Plan* p) {
    // systems below ~2.4M beads: four tiles per SM (measured best over the 256-system mix
    // against two and six per SM with 4-warp CTAs), the last of each architecture a part:
    // one tile more than that is a second round of blocks
    const int sms = sm_count();
    int64_t n_used = 0;
    for (const ArchHost& A : archs) n_used += A.n_chains > 0;
    const int64_t rounds = std::max<int64_t>(1, 4 * sms - n_used);
    const int64_t target_small = (n_beads + rounds - 1) / rounds;
    const size_t first_tile = p->move.size();
    const size_t first_field = p->field.size();
    p->cells32 = p->cells32 && n_cells * spec.n_types < (1ll << 31);
    p->position_bytes += (size_t)n_beads * 12;
    p->cells.push_back({d_sys, n_cells});
    p->cells4 = p->cells4 && spec.n_types <= 3 && spec.p.count_bits == 32 && n_cells % 4 == 0;
    if (p->close.empty()) {
        p->seed = spec.p.seed;
        p->sweep = sweep;
    } else {
        if (p->seed != spec.p.seed) p->one_seed = false;
        if ((p->seed >> 32) != (spec.p.seed >> 32)) p->one_seed_hi = false;
    }
    for (size_t a = 0; a < archs.size(); ++a) {
        const ArchHost& A = archs[a];
        if (A.n_chains == 0) continue;
        int cpt = t.beads_per_tile > 0 ? std::max(1, t.beads_per_tile / A.length) : t.chains_per_tile;
        if (cpt <= 0) {
            const int64_t target = std::min<int64_t>(4096, std::max<int64_t>(A.length, target_small));
            cpt = (int)std::max<int64_t>(1, target / A.length);
            if (cpt >= 8 && cpt * A.length < target) ++cpt;  // of a few long chains a tile more would be too large
            // a few hundred beads at least, so that small systems do not fall into tiles of single chains
            if (A.linear && A.length <= 64) cpt = std::max(cpt, 256 / A.length);
        }
        cpt = std::max(1, std::min(cpt, kMaxTileBeads / A.length));
        for (int c = 0; c < A.n_chains; c += cpt) {
            MoveTile mt;
            mt.sys = d_sys;
            mt.arch = d_arch + a;
            mt.chain0 = A.chain_base + c;
            mt.n_chains = std::min(cpt, A.n_chains - c);
            mt.bead0 = A.bead_base + (int64_t)c * A.length;
            mt.n_tiles_sys = 0;
            mt.arch_index = (int32_t)a;
            p->move.push_back(mt);
            p->max_tile_beads = std::max(p->max_tile_beads, mt.n_chains * A.length);
        }
        p->max_length = std::max(p->max_length, A.length);
        // a bead without bonds has no energy to screen by
        p->chains.push_back({d_sys, d_arch + a, A.length, A.n_chains, A.linear, A.bead_base, A.max_deg ? sweep.screen.on : kScreenOff});
        p->max_deg = std::max(p->max_deg, A.max_deg);
        p->linear = p->linear && A.linear;
    }
    for (size_t i = first_tile; i < p->move.size(); ++i) p->move[i].n_tiles_sys = (int32_t)(p->move.size() - first_tile);
    int64_t cpt_cells = t.cells_per_tile;
    if (cpt_cells <= 0) cpt_cells = std::min<int64_t>(8192, std::max<int64_t>(1024, n_cells / (4 * sms)));
    cpt_cells = (cpt_cells + 3) & ~(int64_t)3;
    const int ntile = (int)((n_cells + cpt_cells - 1) / cpt_cells);
    for (int i = 0; i < ntile; ++i) {
        FieldTile ft;
        ft.sys = d_sys;
        ft.cell0 = (int64_t)i * cpt_cells;
        ft.n_cells = (int)std::min<int64_t>(cpt_cells, n_cells - ft.cell0);
        ft.n_tiles_sys = ntile;
        ft.first_tile = (int32_t)first_field;
        ft.pad = 0;
        p->field.push_back(ft);
    }
    SysClose cl;
    cl.sys = d_sys;
    cl.move_first = (int32_t)first_tile;
    cl.move_count = (int32_t)(p->move.size() - first_tile);
    cl.field_first = (int32_t)first_field;
    cl.field_count = (int32_t)(p->field.size() - first_field);
    p->close.push_back(cl);
    if (p->n_types_uniform == 0 && p->field.size() == (size_t)ntile) p->n_types_uniform = spec.n_types;
    else if (p->n_types_uniform != spec.n_types) p->n_types_uniform = 0;
    // round the smem tile up so float4 staging stays aligned
    p->max_tile_beads = (p->max_tile_beads + 3) & ~3;
    return SCMF_OK;
}

