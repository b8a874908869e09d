"""How the kernels' Python callers keep and choose what they hand to a launch, with the launch itself replaced (no GPU)."""
import types
import weakref

import pytest
import torch

from hipinfer_b200.kernels import library, ops


@pytest.fixture
def launches(monkeypatch):
    """The calls that would have been launches, with what torch.empty made for each and whether it was still held then."""
    calls, made = [], []

    def call(lib, name, *args):
        calls.append(types.SimpleNamespace(name=name, args=args, held=[r() is not None for r, _ in made], buffers=[p for _, p in made]))

    real = torch.empty

    def empty(*size, **kw):
        t = real(*size, **kw)
        made.append((weakref.ref(t), t.data_ptr()))
        return t

    def workspace(M, N, K):
        return 4 * M * N

    fake = types.SimpleNamespace(hb_gemm_simt_workspace=workspace)
    monkeypatch.setattr(ops, "_call", call)
    monkeypatch.setattr(ops, "_need_cuda", lambda *t: None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(library, "load", lambda name: fake)
    monkeypatch.setattr(torch, "empty", empty)
    return calls


def products():
    a, w, out, x = torch.ones(20, 32), torch.ones(48, 32), torch.zeros(20, 48), torch.zeros(20, 48)
    yield lambda: ops.gemm_plain(a, w, out)
    yield lambda: ops.linear_scaled_add(a, ops.Weight(w), x, torch.ones(48))


@pytest.mark.parametrize("which", [0, 1])
def test_a_plain_product_holds_its_workspace_until_it_is_launched(launches, which):
    """A buffer given back before the launch may be another thread's by then, or unmapped."""
    list(products())[which]()
    assert len(launches) == 1 and launches[0].buffers and launches[0].buffers[-1] in launches[0].args and launches[0].held[-1]


@pytest.mark.parametrize("which", [0, 1])
def test_a_plain_product_runs_unsplit_where_no_memory_is_left(launches, which, monkeypatch):
    """The workspace is for speed alone: without one the kernel gives the same bits."""
    def none_left(*size, **kw):
        raise torch.OutOfMemoryError("CUDA out of memory")

    run = list(products())[which]
    counted = library.launches[0]
    monkeypatch.setattr(torch, "empty", none_left)
    run()
    assert len(launches) == 1 and launches[0].args[-2] is None and library.launches[0] == counted
