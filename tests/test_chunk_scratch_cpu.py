"""What the mixers with chunks say about their step buffers: the chunks' part where they may run, and nothing for it where they cannot (float32 models
and sizes that the kernels do not take), since the engine keeps that much memory from the cache."""
import pytest
import torch

from arle_b200 import ops
from arle_b200.parts.delta_rule import GatedDeltaRule, GatedDeltaRuleSpec
from arle_b200.parts.mamba2 import Mamba2, Mamba2Spec


def _loaded(part, dtype):
    part.load({d.name: torch.zeros(d.shape) for d in part.weight_decls()}, dtype, "cpu")
    return part


def _delta(dtype, key_dim=128, value_dim=16, heads=4):
    return _loaded(GatedDeltaRule(GatedDeltaRuleSpec("", 32, heads, 2, key_dim, value_dim, 4, 1e-6)), dtype)


def _mamba2(dtype, state_dim=128, head_dim=16, heads=4):
    return _loaded(Mamba2(Mamba2Spec("", 32, heads, head_dim, state_dim, 2, 4, 1, 1e-6)), dtype)


@pytest.mark.parametrize("make,names", [(_delta, ("key_dim", "value_dim")), (_mamba2, ("state_dim", "head_dim"))], ids=["delta", "mamba2"])
def test_only_what_may_run_is_counted(make, names):
    def per_token(dtype, **kw):
        return make(dtype, **kw).scratch_elements_per_token()

    assert per_token(torch.bfloat16) > per_token(torch.float32) + 1000
    for kw in ({names[0]: 64}, {names[1]: 12}):
        assert per_token(torch.bfloat16, **kw) == per_token(torch.float32, **kw)


def test_the_chunks_fit():
    for make, need in ((_delta, lambda T, R, H: ops.delta_scan_scratch(T, R, H)),
                       (_mamba2, lambda T, R, H: min(T // 32, T // 64 + min(R, T // (ops.DECAY_TC_LONGEST + 1))) * H * 4096)):
        part, other = make(torch.bfloat16), make(torch.float32)
        counted = part.scratch_elements_per_token() - other.scratch_elements_per_token()          # of two bytes
        for T in (64, 80, 159, 160, 192, 1999, 2048, 16384):
            for R in (1, 2, 3, 25, 200):
                assert 2 * need(T, R, part.spec.num_heads) <= T * counted
