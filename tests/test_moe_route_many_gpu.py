"""Routing of thousands of tokens (four or eight tokens per block) equals the routing of a few at a time (one block per token), bit for bit."""
import pytest
import torch

from tests.test_prompt_attention_gpu import DEV, nsq  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,outputs,top,groups,keep", [(1199, 8, 2, 4, 2), (1201, 5, 5, 5, 5), (2499, 31, 3, 1, 1), (2501, 16, 4, 4, 2), (2503, 63, 4, 7, 3), (7001, 64, 8, 8, 4)])
@pytest.mark.parametrize("width,dt", [(136, torch.bfloat16), (50, torch.float32)])
def test_thousands_of_tokens_equal_a_few(nsq, tokens, outputs, top, groups, keep, width, dt):  # noqa: F811
    g = torch.Generator(device=DEV).manual_seed(outputs + width)
    h = torch.randn(tokens, width, generator=g, device=DEV).to(dt)
    w = (torch.randn(outputs, width, generator=g, device=DEV) * width ** -0.5).to(dt)
    gate, corr = torch.randn(width, generator=g, device=DEV).to(dt), torch.randn(outputs, generator=g, device=DEV)
    got = nsq.moe_route(h, w, corr, gate, top, groups, keep, renorm=True)
    few = [nsq.moe_route(h[a:a + 63], w, corr, gate, top, groups, keep, renorm=True) for a in range(0, tokens, 63)]
    for part, alone in zip(got, zip(*few)):
        assert torch.equal(part, torch.cat(alone))
