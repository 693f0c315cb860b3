"""Where the training calls put their results, and without host memory of their own."""

from __future__ import annotations

import shutil
import subprocess

import pytest

from test_c_abi import LIBDIR, ROOT

pytestmark = pytest.mark.gpu


_NO_MEMORY = r"""
#include <vct.h>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>
static bool full = false;
void* operator new(std::size_t n) {
    void* p = full && n > 10000 ? nullptr : std::malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main() {
    vct_mlp* m = nullptr;
    if (vct_mlp_create(0, 1, &m) != VCT_OK) return 1;
    static float a[VCT_MLP_PARAMS], b[VCT_MLP_PARAMS];
    if (vct_mlp_get_params(m, a, VCT_MLP_PARAMS, nullptr) != VCT_OK) return 2;
    full = true;
    if (vct_mlp_get_params(m, b, VCT_MLP_PARAMS, nullptr) != VCT_OK) return 3;
    full = false;
    for (int i = 0; i < VCT_MLP_PARAMS; ++i)
        if (a[i] != b[i]) return 4;
    vct_mlp_destroy(m);
    puts("ok");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_no_exception_leaves_get_params(tmp_path):
    """With no host memory for a staging copy (a program's own operator new throws)."""
    src, exe = tmp_path / "full.cpp", str(tmp_path / "full")
    src.write_text(_NO_MEMORY)
    subprocess.run(["g++", "-std=c++17", "-I", ROOT + "/include", str(src), "-L", LIBDIR, "-lvct", "-Wl,-rpath," + LIBDIR,
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "ok" in r.stdout, (r.returncode, r.stderr)
