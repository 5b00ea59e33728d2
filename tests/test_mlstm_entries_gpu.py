"""The matrix-memory recurrence with its chunks side by side: the entries of a step may come in any order, whatever the order of their rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16 = torch.device("cuda:0"), torch.bfloat16


def scan(lens, H, D, V, order=None, before=None):
    """One step over entries of `lens` tokens that continue stored states; `order`: the order in which the entries are described."""
    from promptcache_b200 import _native_seq as nsq
    g = torch.Generator(device=DEV).manual_seed(D)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    T, B = sum(lens), len(lens)
    proj, offs = rnd(T, 2 * H * D + 2 * H * V).to(BF16), (0, H * D, 2 * H * D, 2 * H * D + H * V)
    ig, fg, w = rnd(T, H), torch.nn.functional.logsigmoid(rnd(T, H) + 3), rnd(H * V).to(BF16)
    s, n, m, out = rnd(B, H, D, V), rnd(B, H, D), rnd(B, H), torch.full((T, H * V), 7.0, device=DEV, dtype=BF16)
    batch = nsq.Batch(range(B), [5] * B, lens, DEV)
    if order is not None:
        for name in ("seq_slot", "seq_pos0", "seq_len", "seq_off"):
            setattr(batch, name, getattr(batch, name)[order].contiguous())
    if before is not None:
        before()
    nsq.mlstm_scan(proj, offs, ig, fg, w, out, s, n, m, 1e-5, batch)
    return out, s, n, m


@pytest.mark.parametrize("lens,H,D,V", [((300, 100, 193, 1, 700), 2, 64, 128), (tuple(range(180, 220)), 1, 16, 40)])
def test_entries_in_any_order(lens, H, D, V):
    order = torch.randperm(len(lens), generator=torch.Generator().manual_seed(1)).flip(0).to(DEV)
    for a, b in zip(scan(lens, H, D, V), scan(lens, H, D, V, order)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lens,V", [((300, 65), 128), ((500,), 512)])
def test_no_room_for_the_chunks_side_by_side(monkeypatch, lens, V):
    """Where their states find no memory, or more than the limit, the chunks run one after the other."""
    from promptcache_b200 import _native_seq as nsq
    empty, refused = torch.empty, []

    def no_room(n, *a, **k):
        if isinstance(n, int) and n == wanted:
            refused.append(n)
            raise torch.OutOfMemoryError("no room")
        return empty(n, *a, **k)
    wanted = int(nsq.load().pcs_mlstm_scratch_floats(sum(lens), len(lens), 1, 64, V))
    ref = scan(lens, 1, 64, V)
    monkeypatch.setattr(nsq, "MLSTM_SCRATCH_MAX", wanted - 1)
    beyond = scan(lens, 1, 64, V)
    monkeypatch.setattr(nsq, "MLSTM_SCRATCH_MAX", wanted)
    short = scan(lens, 1, 64, V, before=lambda: monkeypatch.setattr(nsq.torch, "empty", no_room))
    monkeypatch.setattr(nsq.torch, "empty", empty)
    assert refused
    for a, b, c in zip(ref, beyond, short):
        assert torch.equal(b, c)
        # two forms of one recurrence: sums of up to 64 products in another order, weights and states of 16 bits, results rounded to bfloat16
        assert float((a.float() - b.float()).abs().max()) <= (2.0 ** -7 if a.dtype == BF16 else 2.0 ** -14) * float(a.float().abs().max())
