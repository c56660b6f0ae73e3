"""What a latent attention layer says about its step buffers covers what the built form may hold, however few tokens have long contexts."""
import torch

from arle_b200 import ops
from arle_b200.parts.latent_attention import LatentAttention, LatentAttentionSpec
from arle_b200.parts.base import Part


def test_buffers_of_long_contexts_are_counted():
    H, dn, dr, rank = 4, 64, 32, 128
    spec = LatentAttentionSpec(prefix="", hidden_size=64, num_heads=H, nope_dim=dn, rope_dim=dr, value_dim=dn, kv_rank=rank, scale=0.1, norm_eps=1e-6,
                               position=None)
    part = LatentAttention(spec)
    assert part.scratch_elements_at_least() == 0                     # nothing is built in float32
    part.load({d.name: torch.zeros(d.shape) for d in part.weight_decls()}, torch.bfloat16, "cpu")
    for tokens in (64, 2048, 100_000):
        held = part.scratch_elements_at_least() + tokens * part.scratch_elements_per_token()
        most = max(ops.LATENT_BUILT_MOST * tokens, ops.LATENT_BUILT_PLACES)
        for places in (64, 4096, most // 2, most):                   # the heads that are built at a time, as latent_prefill takes them
            heads = min(H, max(tokens * H // places, ops.LATENT_BUILT_NUMBERS // (places * dn), 1))
            assert places * (rank + dr) + places * 2 * heads * dn <= held
    assert Part.scratch_elements_at_least(part) == 0
