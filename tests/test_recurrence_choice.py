"""Which form of a linear recurrence a layer takes (parts/linear_recurrence.py, parts/retention.py)."""
import pytest
import torch

from gollmgo_b200.csrc import ops
from gollmgo_b200.parts import BuildContext, PartSpec, build_mixer

MIXERS = {
    "mamba2": dict(hidden_size=64, num_heads=4, v_head_dim=32, state=128, groups=2, conv=4, norm_groups=2, eps=1e-6),
    "mlstm": dict(hidden_size=64, num_heads=2, head_dim=128, v_head_dim=64, gate_cap=15.0, eps=1e-6),
    "retention": dict(hidden_size=64, num_heads=2, head_dim=128, v_head_dim=64, decay=[0.9, 0.99], eps=1e-6,
                      position=PartSpec("rope", dict(head_dim=128, theta=10000.0))),
}


def mixer(kind, dtype, device="cpu", max_tokens=2048, max_seqs=16):
    ctx = BuildContext(dtype, device, max_tokens=max_tokens, max_seqs=max_seqs, page_size=16)
    return build_mixer(PartSpec(kind, MIXERS[kind]), ctx), ctx


def chunk_lists(part):
    return [t for t in part.query_tiles() if t.height == ops.LINEAR_CHUNK]


@pytest.mark.parametrize("kind", sorted(MIXERS))
def test_models_in_float32_keep_float32_products(kind):
    assert chunk_lists(mixer(kind, torch.bfloat16)[0])
    assert not chunk_lists(mixer(kind, torch.float32)[0])
