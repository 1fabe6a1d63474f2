"""The measured cases' evaluation in 64 bits stays what the engine computes: a short case of every kind and design, within the
tolerance that the cases state."""

import pytest
import torch

pytestmark = pytest.mark.gpu

SHORT = [
    {"kind": "generate", "shape": "tiny_b", "dtype": "float32", "requests": 2, "prompt": 30, "new": 4},
    {"kind": "prompts", "shape": "tiny_a", "dtype": "float32", "requests": 3, "prompt": 40, "new": 2},
    {"kind": "step", "shape": "7b", "layers": 1, "dtype": "float32", "decodes": 2, "context": 70, "portion": 9, "after": 33},
    {"kind": "step", "shape": "7b", "layers": 1, "dtype": "bfloat16", "decodes": 2, "context": 70, "portion": 65, "after": 33},
    {"kind": "prompts", "shape": "modovik", "dtype": "bfloat16", "requests": 2, "prompt": 40, "new": 2},
    {"kind": "prompts", "shape": "pivinex", "dtype": "bfloat16", "requests": 2, "prompt": 40, "new": 2},
]


@pytest.mark.parametrize("case", SHORT, ids=lambda c: f"{c['kind']}-{c['shape']}-{c['dtype']}")
def test_evaluation_in_64_bits(case):
    from perf import cases
    got, want = cases.run(cases.prepare(case, 3)), cases.exact(case, 3)
    if "ids" in got:
        assert all(torch.equal(a.cpu(), b.cpu()) for a, b in zip(got["ids"], want["ids"]))

    def flat(out):
        rows = out["logits"] if isinstance(out["logits"], (list, tuple)) else [out["logits"]]
        return torch.cat([torch.as_tensor(r).double().cpu().flatten() for r in rows])
    a, b = flat(got), flat(want)
    assert float((a - b).norm() / b.norm()) <= cases.tolerance(case)["rel"]
    torch.cuda.empty_cache()
