"""A decode step replayed from a graph, where every kernel starts as early as it may, against the same step called eagerly."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("method,batch", [("blast", 1), ("blast", 4), ("blast", 16), ("blast_int8", 1), ("blast_int8", 4)])
def test_step_from_a_graph_has_the_bits_of_the_eager_one(method, batch):
    """Widths of the decoder in use: the kernels have to be long enough for the next one to start beside them.  (Not the batches whose down projection goes
    to the cluster kernel, which adds in no fixed order.)"""
    from mem_efficient_blr_b200 import networks as nw
    shape = nw.LlamaShape(layers=3, vocab=1000)
    m = nw.LlamaDecoder(shape, method, batch=batch, cache_len=256, dtype=torch.float16, seed=3, init_on_device=True)
    for c in m.kcache + m.vcache:
        c.normal_(0, 0.5)
    ids = torch.randint(0, shape.vocab, (batch, 1), device=DEV)
    pos = torch.tensor([200], device=DEV)
    step = nw.GraphedCall(m.decode_step, ids.clone(), pos.clone())
    want = m.decode_step(ids, pos).clone()
    caches = [c.clone() for c in m.kcache + m.vcache]
    torch.cuda.synchronize()
    for _ in range(5):
        for c in m.kcache + m.vcache:
            c[:, :, 200] = 7.
        got = step(ids, pos)
        torch.cuda.synchronize()
        assert torch.equal(got, want) and all(torch.equal(a, b) for a, b in zip(caches, m.kcache + m.vcache))
