"""The attention kernels of the slot pool on every device of a process: what they ask of a device is set up on each."""
import pytest
import torch

from tests.test_attention_bias_table_gpu import BF16, F32, nsq  # noqa: F401  (nsq: the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("new,D", [(1, 256), (40, 128)])
def test_every_device(nsq, dt, new, D):  # noqa: F811
    """(The same numbers everywhere; a kernel that was set up on the first device alone cannot be launched on the others.)"""
    g = torch.Generator().manual_seed(new)
    q, k, v = (torch.randn(*s, generator=g).to(dt) for s in ((new, 8 * D), (1, 1, 1024, D), (1, 1, 1024, 128)))
    outs = []
    for i in range(torch.cuda.device_count()):
        dev = torch.device("cuda", i)
        with torch.cuda.device(dev):
            out = torch.full((new, 8 * 128), 7.0, device=dev, dtype=dt)
            nsq.attention(q.to(dev), k.to(dev), v.to(dev), out, 8, D ** -0.5, None, None, False, nsq.Batch([0], [900], [new], dev),
                          workspace=nsq.attn_workspace(new, 8, 128, dev), max_keys=1024)
            outs.append(out.cpu())
    assert bool((outs[0] != 7.0).all()) and all(torch.equal(outs[0], o) for o in outs)
