"""32-bit products that the plain kernel refuses never reach the split kernel: it takes pointers and sizes as they are."""
import pytest
import torch

from hipinfer_b200.kernels import fast, ops


@pytest.fixture
def no_launch(monkeypatch):
    def launched(*_):
        raise AssertionError("launched")
    monkeypatch.setattr(fast, "gemm_split", launched)


def test_tensors_of_the_host_are_refused(no_launch):
    a, w, out = torch.zeros(16, 512), ops.Weight(torch.zeros(512, 512)), torch.zeros(16, 512)
    with pytest.raises(ops.KernelError, match="CUDA tensors only"):
        ops.linear(a, w, out)


@pytest.mark.gpu
@pytest.mark.parametrize("a,w,out,error", [
    ((16, 512), (512, 256), (16, 512), AssertionError),          # K of the weights, shorter and longer
    ((16, 512), (512, 1024), (16, 512), AssertionError),
    ((16, 512), (512, 512), (12, 512), AssertionError),          # an output of fewer rows, of fewer columns, of more
    ((16, 512), (512, 512), (16, 256), AssertionError),
    ((16, 512), (512, 512), (16, 1024), AssertionError),
    ((512,), (512, 512), (512, 512), ops.KernelError),           # rows that are no matrix
])
def test_sizes_that_do_not_match_are_refused(no_launch, a, w, out, error):
    t = lambda s: torch.zeros(*s, device="cuda:0")
    with pytest.raises(error):
        ops.linear(t(a), ops.Weight(t(w)), t(out))


@pytest.mark.gpu
@pytest.mark.parametrize("host", ["a", "w", "out"])
def test_one_tensor_of_the_host_is_refused(no_launch, host):
    a, w, out = (torch.zeros(16, 512, device="cpu" if host == n else "cuda:0") if n != "w" else
                 torch.zeros(512, 512, device="cpu" if host == n else "cuda:0") for n in ("a", "w", "out"))
    with pytest.raises(ops.KernelError, match="CUDA tensors only"):
        ops.linear(a, ops.Weight(w), out)
