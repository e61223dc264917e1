"""A wait between CTAs of one launch that nothing ends gives up and reports it.

The projection's team kernel is launched with half a team: one CTA of a block
that asks for two.  Its first wait has to run out after the two seconds that
wait.cuh allows, set the error flag and leave the kernel with the context
usable; with the flag already set (another team's wait ran out) it has to leave
at once.  The driver is compiled against the library here."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "v2rdm_casscf_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

DRIVER = r"""
#include <chrono>
#include <cstdio>
#include "kernels.cuh"

template <class T>
static T* device(size_t n) {
    void* p = nullptr;
    if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess || cudaMemset(p, 0, n * sizeof(T)) != cudaSuccess) throw 1;
    return static_cast<T*>(p);
}

int main() {
    using namespace v2g;
    const int n = 65, np = 128;
    BlockTask task{};
    task.n = n;
    task.np = np;
    const SignTeam team{0, 0, 2, 0};  // the CTA of rank 1 is missing
    BlockTask* tasks = device<BlockTask>(1);
    SignTeam* teams = device<SignTeam>(1);
    cudaMemcpy(tasks, &task, sizeof task, cudaMemcpyHostToDevice);
    cudaMemcpy(teams, &team, sizeof team, cudaMemcpyHostToDevice);
    double *aty = device<double>(n * n), *c = device<double>(n * n), *x = device<double>(n * n),
           *z = device<double>(n * n), *mu = device<double>(1), *part = device<double>(4), *w[4];
    for (auto& p : w) p = device<double>(np * np);
    unsigned int* bar = device<unsigned int>(1);
    int *hint = device<int>(1), *err = device<int>(1);
    for (int set : {1, 0, 1}) {  // the first also loads the kernel
        cudaMemcpy(err, &set, sizeof set, cudaMemcpyHostToDevice);
        cudaDeviceSynchronize();
        const auto t0 = std::chrono::steady_clock::now();
        cudaError_t e = launch_team_sign(tasks, 1, teams, 1, 1, 1, aty, c, x, z, mu, nullptr, nullptr, w[0], w[1], w[2],
                                         w[3], part, bar, hint, err, 0);
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
        const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        int got = -1;
        cudaMemcpy(&got, err, sizeof got, cudaMemcpyDeviceToHost);
        std::printf("%d %d %.3f\n", (int)e, got, s);
    }
}
"""


def test_wait_of_half_a_team(v2g, tmp_path):
    (tmp_path / "half.cpp").write_text(DRIVER)
    lib = os.path.join(PACKAGE, "lib")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(PACKAGE, "csrc"), "-I", os.path.join(CUDA, "include"),
                    str(tmp_path / "half.cpp"), "-o", str(tmp_path / "half"), "-L", lib, "-lv2rdm_b200",
                    "-Wl,-rpath," + lib, "-L", os.path.join(CUDA, "lib64"), "-lcudart",
                    "-Wl,-rpath," + os.path.join(CUDA, "lib64")], check=True)
    out = subprocess.run([str(tmp_path / "half")], check=True, capture_output=True, text=True, timeout=60).stdout
    rows = [[float(v) for v in k.split()] for k in out.split("\n") if k]
    assert [r[:2] for r in rows] == [[0, 1]] * 3
    s0, s1 = rows[1][2], rows[2][2]
    assert 1.9 <= s0 <= 4.0
    assert s1 <= 0.5
