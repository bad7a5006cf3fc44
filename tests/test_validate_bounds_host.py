"""validate_kernel (csrc/peel.cu) on the host: its source is compiled by the
C++ compiler with one thread standing for the grid, and its arrays end where an
unmapped page begins, so a read past any of them ends the process.  Row
pointers past the number of edges must be refused without reading there."""
import os
import shutil
import subprocess

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tdtdecomposition_gb300", "csrc",
                   "peel.cu")
CXX = shutil.which("g++") or shutil.which("c++")

HEAD = r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <sys/mman.h>
#include <unistd.h>
#define __global__ static
#define __device__ static
#define __forceinline__ inline
#define __restrict__
struct Dim { unsigned x; };
static const Dim blockIdx{0}, threadIdx{0}, blockDim{1}, gridDim{1};
enum { TDT_OK = 0, TDT_ERR_INVALID = 1, TDT_ERR_NOT_ORIENTED = 7 };
struct GridCtl { int status; };
struct PeelCtl { GridCtl g; };
static int atomicMax(int* p, int v) { int o = *p; if (v > o) *p = v; return o; }
"""

MAIN = r"""
template <class T> static T* at_page_end(const T* x, size_t n) {
    const size_t pg = (size_t)sysconf(_SC_PAGESIZE), len = (n * sizeof(T) + pg - 1) / pg * pg;
    char* p = (char*)mmap(nullptr, len + pg, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    mprotect(p + len, pg, PROT_NONE);
    T* d = (T*)(p + len) - n;
    memcpy(d, x, n * sizeof(T));
    return d;
}
int main() {
    // a path 0 -> 1 -> 2 -> 3 with a chord; the last row pointers of each case
    const int32_t rows[4] = {0, 0, 1, 2}, cols[4] = {1, 2, 2, 3};
    const int64_t rps[5][5] = {{0, 2, 3, 4, 4}, {0, 2, 3, 5, 5}, {0, 2, 3, 1000000, 4}, {0, 2, 3, 4, 5}, {0, 2, 9, 9, 4}};
    for (int i = 0; i < 5; i++) {
        PeelCtl c{};
        validate_kernel(at_page_end(rps[i], 5), at_page_end(rows, 4), at_page_end(cols, 4), 4, 4, &c);
        printf("%d ", c.g.status);
    }
    return 0;
}
"""


@pytest.mark.skipif(CXX is None, reason="no C++ compiler")
def test_row_pointers_past_the_edges(tmp_path):
    src = open(SRC).read()
    body = src[src.index("__device__ __forceinline__ int validate_edge("):src.index("// The same when the caller gave no rows")]
    f = tmp_path / "v.cpp"
    f.write_text(HEAD + body + MAIN)
    exe = str(tmp_path / "v")
    subprocess.run([CXX, "-O0", "-std=c++17", "-o", exe, str(f)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, "read past an array (signal %d) after: %s" % (-r.returncode, r.stdout)
    assert r.stdout.split() == ["0", "1", "1", "1", "1"]
