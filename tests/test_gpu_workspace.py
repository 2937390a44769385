"""The workspaces of fmf_dev_csf_fused (FP64) and solphi_mthinc1_: calls on two streams, one
right behind the other, and calls inside a caller's stream capture, give what the same
calls give one at a time, bit for bit."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from fmf import capi
from fmf import config as C

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _phi(torch, shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(shape, dtype=torch.float64, device="cuda", generator=g)


def _csf(L, size, phi, out):
    ni, nj, nk = size
    args = [2.0 / ni, 1.0 / nj, 1.0 / nk, 10.0, 1.0, 1.0] + [ctypes.c_void_p(t.data_ptr()) for t in [phi] + out]
    return L.fmf_dev_csf_fused(capi.FMF_FP64, ni, nj, nk, *args)


def _fields(torch, size, n=3):
    shape = (size[2] + 6, size[1] + 6, size[0] + 6)
    return [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(n)]


@pytest.fixture
def L(fmf_lib):
    yield fmf_lib
    fmf_lib.fmf_set_stream(None)
    fmf_lib.fmf_reset()


@pytest.mark.parametrize("own", [False, True], ids=["callers", "library"])
def test_csf_on_two_streams(L, own):
    """Both streams busy at once (the callers', or the library's own and a caller's): the
    larger grid's kernels run while the smaller's start."""
    torch = pytest.importorskip("torch")
    sizes = [(128, 128, 128), (64, 64, 64)]
    phis = [_phi(torch, (s[2] + 6, s[1] + 6, s[0] + 6), q) for q, s in enumerate(sizes)]
    want = [_fields(torch, s) for s in sizes]
    for s, phi, out in zip(sizes, phis, want):
        assert _csf(L, s, phi, out) == 0
        L.fmf_device_synchronize()
    streams = [torch.cuda.Stream() for _ in sizes]
    got = [[_fields(torch, s) for s in sizes] for _ in range(6)]
    torch.cuda.synchronize()
    for rep in got:
        for q in (0, 1):
            L.fmf_set_stream(None if own and q == 0 else ctypes.c_void_p(streams[q].cuda_stream))
            assert _csf(L, sizes[q], phis[q], rep[q]) == 0
    torch.cuda.synchronize()
    for rep in got:
        for a, b in zip(rep, want):
            assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("own", [False, True], ids=["callers", "library"])
def test_fluxes_on_two_streams(L, own):
    """solphi_mthinc1_ on host arrays that live on the device, each set on its own stream."""
    torch = pytest.importorskip("torch")
    size = (64, 32, 32)
    cfg = C.Config("workspace", *size, 2.0, 1.0, 1.0, dt=1e-3, steps=1)
    rng = np.random.default_rng(2)
    sets = []
    for _ in range(2):
        ins = [rng.uniform(0, 1, cfg.shape)] + [rng.normal(size=cfg.shape) / cfg.dx for _ in range(3)] + \
            [0.2 * cfg.dx / cfg.dt * rng.uniform(-1, 1, cfg.shape) for _ in range(3)]
        ins[1:4] = [a * (rng.uniform(size=cfg.shape) < 0.1) for a in ins[1:4]]
        sets.append((ins, [np.zeros(cfg.shape) for _ in range(3)]))

    def call(q):
        ins, outs = sets[q]
        L.solphi_mthinc1_(*[capi.I(n) for n in size], *[capi.D(1 / d) for d in (cfg.dx, cfg.dy, cfg.dz)],
                          capi.D(cfg.dt), capi.D(2.0), *[capi.P(a) for a in ins + outs])

    def read():
        for _, outs in sets:
            for a in outs:
                L.fmf_sync_to_host(capi.P(a))
        return [a.copy() for _, outs in sets for a in outs]

    for q in (0, 1):
        call(q)
        L.fmf_device_synchronize()
    want = read()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(10):
        for q in (0, 1):
            L.fmf_set_stream(None if own and q == 0 else ctypes.c_void_p(streams[q].cuda_stream))
            call(q)
    torch.cuda.synchronize()
    assert L.fmf_last_error() == 0
    assert all(np.array_equal(a, b) for a, b in zip(read(), want))


CAPTURE = """
import sys
sys.path[:0] = [{tests!r}, {pkg!r}]
import ctypes
import torch
from fmf import capi
from test_gpu_workspace import _csf, _fields, _phi
L = capi.load()
size, larger = (64, 32, 32), (128, 64, 64)
phi, out = _phi(torch, (38, 38, 70), 0), _fields(torch, size)
graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
with torch.cuda.graph(graph, stream=s):  # this process's first call
    L.fmf_set_stream(ctypes.c_void_p(s.cuda_stream))
    assert _csf(L, size, phi, out) == 0
L.fmf_set_stream(None)
plain, aside = [_fields(torch, size) for _ in range(2)]
with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=s):  # and one beside a capture
    torch.zeros(1, device="cuda").add_(1)
    assert _csf(L, size, phi, aside) == 0
assert _csf(L, size, phi, plain) == 0
L.fmf_device_synchronize()
assert _csf(L, larger, _phi(torch, (70, 70, 134), 1), _fields(torch, larger)) == 0
L.fmf_reset()
for _ in range(3):
    for t in out:
        t.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) and torch.equal(a, c) for a, b, c in zip(out, plain, aside))
    assert bool(out[0].abs().max() > 0)
"""


def test_csf_captured(fmf_lib):
    """Captured by the caller as a process's first call, and replayed after a larger call and
    after the kept memory is given back."""
    pytest.importorskip("torch")
    code = CAPTURE.format(tests=os.path.join(ROOT, "tests"), pkg=os.path.join(ROOT, "fel-multi-phase-flow_gb300"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
