"""The shared-memory opt-in of the large kernels (lagrbf_gb300/csrc/lgb_optin.cuh) against a fake of the two runtime calls: each
device of a process opts in, once per kernel; a failure is returned and tried again."""
import os
import subprocess

import lagrbf_gb300

CSRC = os.path.join(os.path.dirname(lagrbf_gb300.__file__), "csrc")

SOURCE = r"""
#include <cstdio>
#include <initializer_list>
#include <thread>
typedef int cudaError_t;
enum { cudaSuccess = 0, cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
static thread_local int device = 0;
static int sets[80], fail = 0, bytes = 0;
static cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
template <typename K> static cudaError_t cudaFuncSetAttribute(K, int, int n)
{
  if (fail) return 98;
  __atomic_fetch_add(&sets[device], 1, __ATOMIC_RELAXED);
  bytes = n;
  return cudaSuccess;
}
#include "lgb_optin.cuh"
static void kernel(int) {}
static int launch() { static unsigned long long done = 0; return lgb_opt_in(kernel, 95000, &done); }
int main()
{
  int bad = 0;
  fail = 1;
  bad += launch() != 98;
  fail = 0;
  for (int r = 0; r < 3; r++)
    for (int d : {0, 1, 7, 63, 70}) { device = d; bad += launch() != 0; }
  std::thread other([&] { device = 5; bad += launch() != 0; });
  other.join();
  printf("%d %d %d %d %d %d %d %d\n", bad, bytes, sets[0], sets[1], sets[7], sets[63], sets[5], sets[70] > 0);
}
"""


def test_every_device_opts_in(tmp_path):
    src = tmp_path / "optin.cpp"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-x", "c++", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(tmp_path / "optin")],
                   check=True)
    out = subprocess.run([str(tmp_path / "optin")], check=True, stdout=subprocess.PIPE, text=True).stdout.split()
    assert list(map(int, out)) == [0, 95000, 1, 1, 1, 1, 1, 1]


def test_no_opt_in_beside_it():
    """Every kernel of the library opts in through the helper."""
    for name in sorted(os.listdir(CSRC)):
        if name.startswith("lgb_") and name != "lgb_optin.cuh":
            with open(os.path.join(CSRC, name)) as f:
                assert "cudaFuncSetAttribute" not in f.read(), name
