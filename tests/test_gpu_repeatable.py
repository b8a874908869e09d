"""The same requests give the same bits, run after run: greedy and drawn tokens, and the logits of prompts in portions and of
decoded rows, in every design and both element types. Kernels start while the one ahead still runs (programmatic dependent
launch); one that reads what the kernel ahead writes before that has ended shows here as bits that change."""
import pytest
import torch

import tiny

pytestmark = pytest.mark.gpu
RUNS = 4


def folder_of(design, which, path):
    if design == "llama":
        return tiny.make_model_folder(path, which, torch.bfloat16)
    import importlib

    return importlib.import_module(f"{design}_models").make_folder(path, which)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("design,which", [("llama", "b"), ("llama", "c"), ("torirax", "r"), ("vegodra", "c"), ("runopel", "c"),
                                          ("mavinex", "c"), ("gakupel", "c"), ("selovik", "c")])
def test_the_same_requests_give_the_same_bits(design, which, dtype, tmp_path):
    from hipinfer_b200 import Engine
    from hipinfer_b200.engine import StepEntry

    made = folder_of(design, which, tmp_path)
    eng = Engine(made if isinstance(made, str) else made[0] if isinstance(made, tuple) else str(made), dtype=dtype, max_batch=4, max_seq=192,
                 max_prefill=96)
    prompts = [tiny.random_tokens(n, eng.vocab, 11 + n) for n in (1, 9, 40, 83)]
    drawn, logits = [], []
    for _ in range(RUNS):
        drawn.append(eng.generate(prompts, 10, temperature=0.9, seed=5))
        rows = []
        for n in (60, 1, 1, 30, 1):          # a prompt in two portions, single rows behind and between
            entries = [StepEntry(r, prompts[3 - r % 2][:n] if n > 1 else [7 + r], [len(prompts[3 - r % 2][:n]) - 1 if n > 1 else 0])
                       for r in range(3)]
            rows.append(eng.runner.step(entries).clone())
        for r in range(3):
            eng.runner.end(r)
        logits.append(torch.cat(rows).cpu())
    eng.close()
    assert all(d == drawn[0] for d in drawn[1:])
    assert all(torch.equal(a, logits[0]) for a in logits[1:])
