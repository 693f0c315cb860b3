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


def test_loss_into_any_memory():
    """The losses of two steps in memory that the update kernel stores to and
    in memory that it must not: pinned and pageable host memory, and a place
    that is not a float's (a copy brings it there, or refuses); then under
    capture."""
    import torch

    torch.manual_seed(1)
    rows, targets = torch.randn(300, 42, device="cuda"), torch.rand(300, 3, device="cuda")
    opt = L.vct_adam(1e-3, 0.9, 0.999, 1e-8)
    want = torch.zeros(2, device="cuda")
    m = api.Mlp(seed=2)
    for k in range(2):
        m.train_step(rows, targets, None, 300, 1e-3, want[k:])
    params = m.params()

    def steps(pointers, stream=0):
        m = api.Mlp(seed=2)
        for p in pointers:
            L.call("vct_mlp_train_step", m.handle, rows.data_ptr(), targets.data_ptr(), 0, 300, C.byref(opt), p, stream)
        torch.cuda.synchronize()
        assert (m.params() == params).all()

    pinned = torch.zeros(2).pin_memory()
    steps([pinned.data_ptr(), pinned.data_ptr() + 4])
    assert torch.equal(pinned, want.cpu())
    odd = torch.zeros(9, dtype=torch.uint8, device="cuda")
    steps([odd.data_ptr() + 1, odd.data_ptr() + 5])
    assert torch.equal(odd[1:].cpu().view(torch.float32), want.cpu())
    steps([0, 0])
    pageable = torch.full((2,), -1.0)
    m = api.Mlp(seed=2)
    for k in range(2):
        try:
            m.train_step(rows, targets, None, 300, 1e-3, pageable.data_ptr() + 4 * k)
        except L.VctError as e:
            assert e.status == L.VCT_ERR_CUDA and pageable[k] == -1.0
    torch.cuda.synchronize()
    assert (m.params() == params).all()
    assert all(p in (-1.0, w) for p, w in zip(pageable.tolist(), want.tolist()))

    m, loss, graph, st = api.Mlp(seed=2), torch.zeros(2, device="cuda"), torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=st):
        for k in range(2):
            m.train_step(rows, targets, None, 300, 1e-3, loss[k:])
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(loss, want) and (m.params() == params).all()


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
