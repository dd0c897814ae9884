"""Batch-invariant mode at the head sizes of real models: a request's bfloat16 logits are the same bit for bit alone and among twenty."""
import pytest
import torch

pytestmark = pytest.mark.gpu
WIDTH, VOCAB, OTHERS = 512, 300, 19


def luzitar():
    linear = {"heads": 8, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** -(3 + h) for h in range(8)]}
    attention = {"heads": 4, "kv_heads": 2, "dim": 64, "vdim": 64, "scale": 0.2, "mask": {"size": 48, "keep_first": 8}, "conv": 4,
                 "rot": {"dims": 32, "base": 10000.0}}
    mlp = {"kind": "moe", "expert": {"ff": 128, "limit": 7.0}, "router": {"experts": 8, "top": 2, "groups": {"count": 4, "keep": 2}}}
    return {"architecture": "Luzitar", "vocab": VOCAB, "width": WIDTH, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
            "layers": [{"type": "lightning", "mixer": linear, "mlp": mlp}, {"type": "attention", "mixer": attention, "mlp": mlp}]}


def pilonex():
    left = {"heads": 4, "kv_heads": 2, "dim": 64, "vdim": 64, "scale": 0.125, "mask": {"size": 48}, "rot": {"dims": 64, "base": 10000.0}}
    right = {"heads": 8, "kv_heads": 4, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 32, "gate_rank": 32}
    mlp = {"kind": "dense", "ff": 256, "limit": 7.0}
    return {"architecture": "Pilonex", "vocab": VOCAB, "width": WIDTH, "norm": {"eps": 1e-6}, "streams": 2,
            "layers": [{"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0}, "mlp": mlp},
                       {"type": "mlstm", "mixer": {"heads": 8, "dim": 128, "vdim": 128, "gate_cap": 15.0}, "mlp": mlp}]}


MAKERS = {"luzitar": luzitar, "pilonex": pilonex}


@pytest.mark.parametrize("name", sorted(MAKERS))
def test_logits_alone_and_among_twenty(name):
    from openinfer_b200 import ModelRunner, StepEntry
    from openinfer_b200.config.base import resolve_architecture
    from openinfer_b200.kernels import policy
    raw = MAKERS[name]()
    config = resolve_architecture(raw).config_cls.from_dict(raw)
    g = torch.Generator().manual_seed(3)
    lens = [43, 1, 30] + [26 + i for i in range(OTHERS - 2)]          # some 700 prompt rows in a step
    tokens = [torch.randint(0, VOCAB, (n + 3,), generator=g).tolist() for n in lens]
    policy.set_batch_invariant(True)
    try:
        runner = ModelRunner.build(config, 5, dtype="bfloat16", page_size=16, max_requests=len(lens), max_tokens=64 * len(lens))

        def run(which):
            rows = {r: [] for r in which}
            steps = [[(r, 0, lens[r]) for r in which]] + [[(r, lens[r] + i, 1) for r in which] for i in range(3)]
            for step in steps:
                out, at = runner.step([StepEntry(r, tokens[r][pos: pos + n], list(range(n))) for r, pos, n in step]), 0
                for r, _, n in step:
                    rows[r].append(out[at: at + n].clone())
                    at += n
            for r in which:
                runner.end(r)
            return {r: torch.cat(v) for r, v in rows.items()}

        together = run(list(range(len(lens))))
        for r in (0, 1, len(lens) - 1):
            assert torch.equal(run([r])[r], together[r]), r
    finally:
        policy.set_batch_invariant(False)
