"""Error words that kernels set on a system reach the caller: from the blocking calls of a
batch, which has many systems, and from the server, which hands out no counts of such a
system.  The words are set from the host, by programs built against the library's own
headers: into a member's record, and by a stand-in for the launch of many sweeps.  And a
launch of many sweeps whose blocks do not wait for one another sets the word, no launch
uses its barrier again, and the system stays where it is while the others of a batch go
on.  Where a context cannot hold the launch's blocks all at once (again a stand-in says so),
sweeps are launched one by one."""
import os
import subprocess

import pytest

import new_arch_b200.build as build

pytestmark = pytest.mark.gpu

COMMON = r"""
#include <chrono>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "scmf_engine.h"
using namespace scmf;
#define WANT(expr, want)                                                                          \
    do {                                                                                          \
        const long long got_ = (long long)(expr), want_ = (long long)(want);                      \
        if (got_ != want_) {                                                                      \
            std::printf("%s is %lld, not %lld (%s)\n", #expr, got_, want_, scmf_last_error());    \
            std::exit(1);                                                                         \
        }                                                                                         \
    } while (0)
static scmf_spec* melt(int chains, int length, int edge, uint64_t seed) {
    scmf_spec* s = nullptr;
    WANT(scmf_spec_create(2, edge, edge, edge, edge, edge, edge, &s), SCMF_OK);
    const double xn[4] = {50, 20, 20, 50};
    WANT(scmf_spec_set_xn(s, xn, 2), SCMF_OK);
    scmf_params p{};
    p.reference_nbeads = length;
    p.harmonic_normb = 3.0;
    p.smc_a = 0.5;
    p.seed = seed;
    p.hamiltonian = SCMF_HAM_SCMF0;
    p.field_rule = SCMF_FIELD_EVERY;
    p.count_bits = 32;
    WANT(scmf_spec_set_params(s, &p), SCMF_OK);
    std::vector<int32_t> type(length), bonds;
    for (int i = 0; i < length; ++i) type[i] = 2 * i >= length;
    for (int i = 0; i + 1 < length; ++i) bonds.insert(bonds.end(), {i, i + 1});
    WANT(scmf_spec_add_arch(s, length, chains, type.data(), length - 1, bonds.data(), 0.4), SCMF_OK);
    return s;
}
static scmf_system* started(scmf_spec* spec) {
    scmf_system* s = nullptr;
    WANT(scmf_system_create(spec, nullptr, &s), SCMF_OK);
    WANT(scmf_init_coords(s), SCMF_OK);
    return s;
}
static void set_word(const SysDev* d, uint32_t v) {
    WANT(cudaMemcpy((char*)d + offsetof(SysDev, error_word), &v, 4, cudaMemcpyHostToDevice), 0);
}
"""

BATCH = COMMON + r"""
int main() {
    scmf_system* s[3];
    for (int i = 0; i < 3; ++i) s[i] = started(melt(200 + 10 * i, 32, 10, 5 + i));
    scmf_batch* b = nullptr;
    WANT(scmf_batch_create(s, 3, nullptr, nullptr, &b), SCMF_OK);
    WANT(scmf_batch_step(b, 2), SCMF_OK);
    set_word(s[1]->d_sys, 8);
    float ms[3];
    scmf_tune tune;
    WANT(scmf_batch_step(b, 2), SCMF_E_DEVICE);
    WANT(scmf_batch_step_profiled(b, 1, ms, ms + 1, ms + 2), SCMF_E_DEVICE);
    WANT(scmf_batch_autotune(b, 1, &tune), SCMF_E_DEVICE);
    WANT(scmf_batch_run(s, 3, 1, nullptr), SCMF_E_DEVICE);
    WANT(scmf_batch_run(s + 2, 1, 1, nullptr), SCMF_OK);
    set_word(s[1]->d_sys, 0);
    WANT(scmf_batch_step(b, 1), SCMF_OK);
    WANT(scmf_batch_autotune(b, 1, &tune), SCMF_OK);
    scmf_batch_destroy(b);
    for (auto* x : s) scmf_system_destroy(x);
    return 0;
}
"""

WAITS = COMMON + r"""
static SysDev record(const scmf_system* s) {
    SysDev d;
    WANT(cudaMemcpy(&d, s->d_sys, sizeof d, cudaMemcpyDeviceToHost), 0);
    return d;
}
static std::vector<uint32_t> counts(const scmf_system* s) {
    std::vector<uint32_t> c((size_t)s->n_cells * 2);
    WANT(scmf_get_counts(s, c.data(), c.size()), SCMF_OK);
    return c;
}
int main() {
    scmf_system* s = started(melt(60000, 32, 64, 5));
    WANT(s->plan.d_run != nullptr, true);  // many sweeps a launch
    s->plan.run.wait = 0;                  // a look or two at the count, and no more
    WANT(scmf_step(s, 20), SCMF_E_DEVICE);
    WANT(record(s).error_word, kErrorBarrier);
    WANT(record(s).step, 0);
    s->plan.run.wait = (uint32_t)(kWaitClocks >> kWaitShift);
    set_word(s->d_sys, 0);  // as if nothing had been: the plan's barrier stays broken
    WANT(scmf_step(s, 1100), SCMF_E_DEVICE);
    WANT(record(s).error_word, kErrorBarrier);
    WANT(record(s).step, 0);
    const auto at = counts(s);
    scmf_system* other = started(melt(400, 32, 12, 6));
    scmf_system* pair[2] = {s, other};
    scmf_batch* b = nullptr;
    WANT(scmf_batch_create(pair, 2, nullptr, nullptr, &b), SCMF_OK);
    WANT(b->plan.d_run != nullptr, true);
    WANT(scmf_batch_step(b, 3), SCMF_E_DEVICE);
    WANT(record(s).step, 0);
    WANT(counts(s) == at, true);
    WANT(record(other).step, 3);
    WANT(record(other).error_word, 0);
    scmf_batch_destroy(b);
    scmf_system* same = started(melt(400, 32, 12, 6));
    WANT(scmf_step(same, 3), SCMF_OK);
    WANT(counts(other) == counts(same), true);
    return 0;
}
"""

SERVER = COMMON + r"""
// in place of the library's: no sweep, the error word of every system
int scmf::launch_run(const LaunchShape&, const RunArgs& run, void* stream) {
    std::vector<RunSystem> systems(run.n_sys);
    WANT(cudaMemcpyAsync(systems.data(), run.systems, systems.size() * sizeof(RunSystem), cudaMemcpyDeviceToHost,
                         (cudaStream_t)stream), 0);
    WANT(cudaStreamSynchronize((cudaStream_t)stream), 0);
    for (const RunSystem& r : systems) set_word(r.sys, 8);
    return 0;
}
int main() {
    scmf_server_opts opts{};
    opts.hbm_budget_bytes = 1ull << 30;
    scmf_server* server = nullptr;
    WANT(scmf_server_create(&opts, &server), SCMF_OK);
    std::vector<uint32_t> counts(2 * 1000, 0xABABABABu);
    uint64_t id = 0;
    WANT(scmf_server_submit(server, melt(200, 32, 10, 5), 3, counts.data(), &id), SCMF_OK);
    scmf_result r{};
    int n = 0;
    for (int i = 0; i < 100 && !n; ++i) WANT(scmf_server_poll(server, &r, 1, &n, 200), SCMF_OK);
    WANT(n, 1);
    WANT(r.id, id);
    WANT(r.status, SCMF_E_DEVICE);
    for (uint32_t c : counts) WANT(c, 0xABABABABu);
    scmf_server_destroy(server);
    return 0;
}
"""


SMALL = COMMON + r"""
// as in a context with a part of the GPU's SMs
static int asked = 0;
int scmf::launch_run(const LaunchShape&, const RunArgs&, void*) {
    ++asked;
    return (int)cudaErrorCooperativeLaunchTooLarge;
}
int main() {
    scmf_system* s[2] = {started(melt(300, 32, 12, 5)), started(melt(300, 32, 12, 5))};
    WANT(s[0]->plan.d_run != nullptr, true);
    WANT(scmf_step(s[0], 7), SCMF_OK);
    WANT(asked, 1);
    for (int i = 0; i < 7; ++i) WANT(scmf_step(s[1], 1), SCMF_OK);
    WANT(asked, 1);
    std::vector<float> x[2];
    scmf_stats st[2];
    for (int i = 0; i < 2; ++i) {
        x[i].resize(s[i]->n_beads * 3);
        WANT(scmf_get_coords(s[i], x[i].data(), x[i].size()), SCMF_OK);
        WANT(scmf_get_sweep_stats(s[i], &st[i]), SCMF_OK);
        WANT(st[i].step, 7);
    }
    WANT(x[0] == x[1], true);
    WANT(st[0].total_accepts, st[1].total_accepts);
    return 0;
}
"""


def _run(tmp_path, program):
    lib = build.LIB
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(program)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", build.INC, "-I", build.CSRC, "-I",
                    os.path.join(build.CUDA, "include"), str(src), "-o", str(exe), "-L", os.path.dirname(lib), "-lscmf",
                    "-Wl,-rpath," + os.path.dirname(lib), "-L", os.path.join(build.CUDA, "lib64"), "-lcudart_static", "-ldl",
                    "-lrt", "-pthread"], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr


def test_batch(tmp_path):
    _run(tmp_path, BATCH)


def test_blocks_that_do_not_wait(tmp_path):
    _run(tmp_path, WAITS)


def test_blocks_that_do_not_fit(tmp_path):
    _run(tmp_path, SMALL)


def test_server(tmp_path):
    _run(tmp_path, SERVER)
