"""The host copies' thread pool on the CPU: bytes of copies of ragged lengths, the time of a chunk where the
threads outnumber the CPUs, and the CPU quota of a control group (fake files)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = r"""
#include "host_copy.cuh"
#include <sched.h>
#include <cstdio>
#include <cstdlib>
namespace hpcs {  // what the rest of the library defines
int fail(int s, const std::string&) { return s; }
int cuda_fail(cudaError_t, const char*) { return 1; }
}
int main(int argc, char** argv) {
  if (argc == 3) {
    std::printf("%d\n", hpcs::quota_cpus(argv[1], argv[2]));
    return 0;
  }
  cpu_set_t set;
  CPU_ZERO(&set);
  cpu_set_t all;
  sched_getaffinity(0, sizeof all, &all);
  for (int i = 0, n = 0; i < CPU_SETSIZE && n < 2; i++)
    if (CPU_ISSET(i, &all)) CPU_SET(i, &set), n++;
  sched_setaffinity(0, sizeof set, &set);
  hpcs::CopyPool pool(7);
  std::vector<unsigned char> src(3 << 20), dst(3 << 20);
  for (size_t i = 0; i < src.size(); i++) src[i] = (unsigned char)(i * 2654435761u >> 13);
  for (size_t n : {size_t(1), size_t(63), size_t(4097), size_t(262144), size_t(1000003), size_t(3 << 20) - 5}) {
    std::fill(dst.begin(), dst.end(), 0);
    pool.copy(dst.data() + 3, src.data() + 1, n);
    if (std::memcmp(dst.data() + 3, src.data() + 1, n) || dst[2] || dst[3 + n]) return 2;
  }
  std::vector<double> us;
  for (int i = 0; i < 200; i++) {
    const auto t0 = std::chrono::steady_clock::now();
    pool.copy(dst.data(), src.data(), size_t(512) << 10);
    us.push_back(std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count());
  }
  std::sort(us.begin(), us.end());
  std::printf("%.1f\n", us[100]);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("pool")
    src, exe = d / "pool.cu", d / "pool"
    src.write_text(SOURCE)
    subprocess.run([NVCC, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(ROOT, "hpcsharp_b200", "csrc"), "-Xcompiler", "-pthread", "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    return str(exe)


def test_copies_with_more_threads_than_cpus(program):
    """8 copying threads on 2 CPUs: a thread that looks for work gives its CPU to one that has some (a 512 KiB
    chunk 27 us; 430 where it does not)."""
    res = subprocess.run([program], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stderr
    assert float(res.stdout) < 200.0


@pytest.mark.parametrize("files,group,want", [
    ({}, "/", 0),
    ({"cpu.max": "max 100000"}, "/", 0),
    ({"cpu.max": "200000 100000"}, "/", 2),
    ({"cpu.max": "max 100000", "a/cpu.max": "300000 100000", "a/b/cpu.max": "max 100000"}, "/a/b", 3),
    ({"a/cpu.max": "800000 100000", "a/b/cpu.max": "150000 100000"}, "/a/b", 2),
    ({"a/cpu.max": "20000 100000"}, "/a", 1),
    ({"cpu/cpu.cfs_quota_us": "400000", "cpu/cpu.cfs_period_us": "100000"}, "/", 4),
    ({"cpu/cpu.cfs_quota_us": "-1", "cpu/cpu.cfs_period_us": "100000"}, "/", 0),
])
def test_quota(program, tmp_path, files, group, want):
    for name, text in files.items():
        p = tmp_path / "fs" / name
        p.parent.mkdir(parents=True, exist_ok=True)
        p.write_text(text + "\n")
    (tmp_path / "fs").mkdir(exist_ok=True)
    (tmp_path / "self").write_text(f"1:cpu:/\n0::{group}\n")
    out = subprocess.run([program, str(tmp_path / "fs"), str(tmp_path / "self")], capture_output=True, text=True, timeout=60)
    assert int(out.stdout) == want
