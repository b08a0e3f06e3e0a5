"""Who waits for whom while large host copies are under way: a system is made and destroyed
beside a copy that holds the staging buffer, and a copy whose stream still has other work to
do does not hold it, so that another copy is staged meanwhile."""
import os
import subprocess

import pytest

import new_arch_b200.build as build

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <future>
#include <thread>
#include <vector>
#include "scmf_engine.h"
using namespace scmf;
static void want(bool ok, const char* what) {
    if (ok) return;
    std::printf("%s\n", what);
    std::fflush(stdout);
    std::_Exit(1);
}
static std::atomic<bool> go{false};
static void hold(void*) {  // a stream's earlier work, for ten seconds at most
    for (int i = 0; i < 1000 && !go; ++i) std::this_thread::sleep_for(std::chrono::milliseconds(10));
}
int main() {
    const size_t bytes = (size_t)96 << 20;
    std::vector<char> a(bytes, 1), b(bytes, 2), back(bytes);
    char *da = nullptr, *db = nullptr;
    cudaStream_t sa, sb;
    want(cudaMalloc((void**)&da, bytes) == 0 && cudaMalloc((void**)&db, bytes) == 0, "memory");
    want(cudaStreamCreateWithFlags(&sa, cudaStreamNonBlocking) == 0, "stream");
    want(cudaStreamCreateWithFlags(&sb, cudaStreamNonBlocking) == 0, "stream");
    stage_system_made();
    scmf_status rc = SCMF_OK;
    bool looked = false;
    const auto during = [&](size_t) -> scmf_status {  // the copy holds the buffer here
        if (!looked) {
            looked = true;
            auto other = std::async(std::launch::async, [] { stage_system_made(); stage_system_gone(); });
            want(other.wait_for(std::chrono::seconds(3)) == std::future_status::ready, "a system waits for a copy");
        }
        return SCMF_OK;
    };
    want(copy_to_device_staged(da, a.data(), bytes, sa, during, &rc) && rc == SCMF_OK && looked, "the first copy");
    want(cudaLaunchHostFunc(sa, hold, nullptr) == 0, "host function");
    auto late = std::async(std::launch::async, [&] {
        scmf_status r = SCMF_OK;
        return copy_to_device_staged(da, b.data(), bytes, sa, nullptr, &r) && r == SCMF_OK;
    });
    std::this_thread::sleep_for(std::chrono::milliseconds(300));
    want(copy_to_device_staged(db, a.data(), bytes, sb, nullptr, &rc) && rc == SCMF_OK, "a copy that waits holds the buffer");
    go = true;
    want(late.get(), "the late copy");
    want(copy_to_host(back.data(), da, bytes, sa) == SCMF_OK && back == b, "what the late copy brought");
    want(copy_to_host(back.data(), db, bytes, sb) == SCMF_OK && back == a, "what the other brought");
    stage_system_gone();
    return 0;
}
"""


def test_locks(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", build.INC, "-I", build.CSRC, "-I",
                    os.path.join(build.CUDA, "include"), str(src), "-o", str(exe), "-L", os.path.dirname(build.LIB), "-lscmf",
                    "-Wl,-rpath," + os.path.dirname(build.LIB), "-L", os.path.join(build.CUDA, "lib64"), "-lcudart_static",
                    "-ldl", "-lrt", "-pthread"], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
