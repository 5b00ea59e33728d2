"""Routing of many tokens (four warps per token, two tokens per block) equals the routing of each token alone (one block per token), bit for bit."""
import pytest
import torch

from tests.test_prompt_attention_gpu import DEV, nsq  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("outputs,top,groups,keep", [(1, 1, 1, 1), (3, 2, 1, 1), (5, 5, 5, 5), (16, 4, 4, 2), (256, 8, 8, 4)])
@pytest.mark.parametrize("tokens,width,dt", [(64, 2048, torch.bfloat16), (65, 1032, torch.bfloat16), (67, 50, torch.float32)])
def test_many_tokens_equal_single_ones(nsq, outputs, top, groups, keep, tokens, width, dt):  # noqa: F811
    g = torch.Generator(device=DEV).manual_seed(outputs + width)
    h = torch.randn(tokens, width, generator=g, device=DEV).to(dt)
    w = (torch.randn(outputs, width, generator=g, device=DEV) * width ** -0.5).to(dt)   # (outputs of order 1: no chosen score underflows, none is 0 / 0)
    gate = torch.randn(width, generator=g, device=DEV).to(dt)
    corr = torch.randn(outputs, generator=g, device=DEV)
    got = nsq.moe_route(h, w, corr, gate, top, groups, keep, renorm=True)
    few = [nsq.moe_route(h[a:a + 33], w, corr, gate, top, groups, keep, renorm=True) for a in range(0, tokens, 33)]   # (under 64 tokens: a block each)
    for part, alone in zip(got, zip(*few)):
        assert torch.equal(part, torch.cat(alone))
