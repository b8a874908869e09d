"""How the kernels' Python callers keep and choose what they hand to a launch, with the launch itself replaced (no GPU)."""
import types
import weakref

import pytest
import torch

from hipinfer_b200.kernels import fast, library, ops


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


@pytest.mark.parametrize("M,N,K,n,cut", [(512, 2048, 2048, 4, True), (700, 2048, 2048, 3, True), (1000, 2048, 2048, 2, False), (128, 1024, 1024, 2, False),
                                         (512, 3072, 3072, 3, True), (700, 3072, 3072, 2, False), (512, 4096, 4096, 2, True), (1000, 2048, 8192, 2, True),
                                         (2048, 4096, 4096, 0, False), (64, 1024, 1024, 2, None), (300, 512, 1536, 3, False)])
def test_products_of_portions_are_cut_along_k_where_that_pays(monkeypatch, M, N, K, n, cut):
    """Both sides of the rule (n: the slices that fit the SM pairs); up to 64 rows the small products' kernel has them."""
    monkeypatch.setattr(fast, "_tc_ok", lambda a, w: True)
    monkeypatch.setattr(fast, "_fn", lambda name: {"hb_gemm_tc_splits": lambda *size: n}[name])
    monkeypatch.setattr(fast, "gemm_tc_slices", lambda a, w: True)
    monkeypatch.setattr(fast, "gemm_stream_slices", lambda a, w: None)
    a, w = torch.empty(M, K, device="meta"), ops.Weight(torch.empty(N, K, device="meta"))
    assert fast.linear_slices(a, w, residual=True) == (cut or None) and fast.linear_slices(a, w) is None


def test_the_plain_kernels_may_be_asked_for_after_the_import():
    """HIPINFER_B200_PLAIN is read when a kernel is first chosen, not when the package is imported."""
    import os
    import subprocess
    import sys

    code = ("import os, hipinfer_b200, hipinfer_b200.engine\nfrom hipinfer_b200.kernels import ops\n"
            "os.environ['HIPINFER_B200_PLAIN'] = '1'\nassert not ops.fast_kernels_on()\n"
            "from hipinfer_b200.kernels import fast\nassert fast.PLAIN_ONLY and ops.fast is fast")
    env = {k: v for k, v in os.environ.items() if k != "HIPINFER_B200_PLAIN"}
    subprocess.run([sys.executable, "-c", code], check=True, env=env, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
