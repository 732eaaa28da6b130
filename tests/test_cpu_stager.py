"""The staged copies (csrc/cgfd_stager.h) against a CUDA runtime of host stand-ins: what they copy, and
what they do where pinned memory is refused."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "cgfd_stager.h"

#include <cstdio>
#include <cstdlib>

static long long g_grants, g_pinned;  // host allocations still granted; bytes granted so far
extern "C" {
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  if (g_grants-- <= 0) return cudaErrorMemoryAllocation;
  g_pinned += (long long)n;
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "refused"; }
}

// argv: grants, then transfers "o:bytes:parts" (out, in parts) or "i:bytes" (in); a line of pinned
// bytes so far after each
int main(int argc, char **argv) {
  g_grants = std::atoll(argv[1]);
  cgfd::PinnedStager &ps = cgfd::PinnedStager::for_device(0);
  for (int a = 2; a < argc; a++) {
    char kind;
    size_t n;
    int parts = 1;
    std::sscanf(argv[a], "%c:%zu:%d", &kind, &n, &parts);
    std::vector<unsigned char> src(n), dst(n * parts + 1, 77);
    auto value = [&](size_t at, int part) { return (unsigned char)(at * 131 + (at >> 9) + part * 29); };
    if (kind == 'o') {
      ps.copy_out(dst.data(), src.data(), n, parts, nullptr, [&](int q) {
        for (size_t t = 0; t < n; t++) src[t] = value(t, q);
      });
    } else {
      for (size_t t = 0; t < n; t++) src[t] = value(t, 0);
      ps.copy(dst.data(), src.data(), n, nullptr);
    }
    for (int q = 0; q < parts; q++)
      for (size_t t = 0; t < n; t++)
        if (dst[(size_t)q * n + t] != value(t, q)) return std::printf("%s: byte %zu of part %d\n", argv[a], t, q), 1;
    if (dst.back() != 77) return std::printf("%s: wrote beyond the end\n", argv[a]), 1;
    std::printf("%lld\n", g_pinned);
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("stager")
    (d / "t.cpp").write_text(PROGRAM)
    exe = str(d / "t")
    subprocess.run(["/usr/bin/g++", "-O1", "-std=c++17", "-fopenmp", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "gpu-cgfd3d-elastic_b200", "csrc"), "-I/usr/local/cuda/include",
                    str(d / "t.cpp"), "-o", exe], check=True)
    return exe


def _run(program, grants, *transfers):
    r = subprocess.run([program, str(grants), *transfers], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return [int(v) for v in r.stdout.split()]


@pytest.mark.parametrize("grants", [0, 1, 2, 100])
def test_transfers_are_whole_with_and_without_pinned_memory(program, grants):
    mib = 1 << 20
    pinned = _run(program, grants, "o:1:3", f"o:{3 * mib + 5}:9", f"i:{64 * mib}", f"o:{64 * mib + 1}:2", "i:0", "o:0:1",
                  f"i:{130 * mib + 7}", f"o:{128 * mib}:1", "i:12345")
    assert (pinned[-1] > 0) == (grants > 0)


def test_short_transfers_take_little_pinned_memory(program):
    """A third of a transfer's bytes, rounded up to a piece of 8 MiB for each of the two chunks, and twice
    64 MiB at most; a later transfer takes what an earlier one had."""
    mib = 1 << 20
    first, second, third, last = _run(program, 100, f"o:{45 * mib}:1", f"o:{20 * mib}:9", f"i:{100 * mib}", f"o:{260 * mib}:2")
    assert first <= 45 * mib / 3 + 2 * 8 * mib
    assert second <= 180 * mib / 3 + 2 * 8 * mib
    assert third == second
    assert last == 128 * mib
