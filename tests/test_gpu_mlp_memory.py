"""Where the training calls put their results: memory of the host, pinned or
not, of the network's device, and places that are not a float's."""

from __future__ import annotations

import ctypes as C
import shutil
import subprocess

import pytest

from test_c_abi import LIBDIR, ROOT
from vct_gb300 import _lib as L
from vct_gb300 import api

pytestmark = pytest.mark.gpu


def _get(m, pointer):
    L.check(L.load().vct_mlp_get_params(m.handle, C.cast(pointer, C.POINTER(C.c_float)), api.Mlp.NPARAMS, 0),
            "vct_mlp_get_params")


def test_parameters_into_any_memory():
    import torch

    m = api.Mlp(seed=2)
    want = torch.from_numpy(m.params())
    assert want.abs().sum() > 0
    pinned, device = torch.zeros(api.Mlp.NPARAMS).pin_memory(), torch.zeros(api.Mlp.NPARAMS, device="cuda")
    _get(m, pinned.data_ptr())
    _get(m, device.data_ptr())
    assert torch.equal(pinned, want) and torch.equal(device.cpu(), want)


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
