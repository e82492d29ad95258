"""The workspace of a stream under several threads: growth by one thread beside calls of another, calls of several threads at once."""
import sys
import threading

import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _together(*work):
    """Runs the functions in threads of their own that start together; raises what one of them raised."""
    errors, start = [], threading.Barrier(len(work))

    def body(f):
        try:
            start.wait()
            f()
        except BaseException as e:  # noqa: BLE001 (handed to the test's thread)
            errors.append(e)

    threads = [threading.Thread(target=body, args=(f,)) for f in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def test_calls_beside_a_growing_workspace():
    """A call must get pointer and size of one buffer while another thread replaces the stream's buffer by a larger one."""
    import mem_efficient_blr_b200.blast_kernels as bk
    from mem_efficient_blr_b200 import _lib as L
    x, U, Vt, S = (t.to(DEV) for t in orc.make_blast_inputs(4, 512, 768, 4, 128, torch.float16, seed=1))
    want = bk.blast_torch_layout(x, U, Vt, S)
    torch.cuda.synchronize()
    for _ in range(8):
        st, grown = torch.cuda.Stream(), threading.Event()

        def call():
            with torch.cuda.stream(st):
                while True:
                    last = grown.is_set()
                    assert torch.equal(bk.blast_torch_layout(x, U, Vt, S), want)
                    if last:
                        break

        def grow():
            try:
                for bits in range(22, 27):   # (a workspace has a fixed head of 2 MiB and 1 KiB)
                    L.workspace(torch.device(DEV), st.cuda_stream, 1 << bits)
            finally:
                grown.set()

        _together(call, grow)


def test_calls_of_two_threads_on_one_stream():
    """The launches of a call hand over in the stream's workspace: those of another thread must not come in between."""
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    import mem_efficient_blr_b200.monarch_kernels as mk

    def layer(seed, N):
        """(call, result) of operators with fixed summation orders, some through the direct calls, some through ctypes."""
        x, U, Vt, S = (t.to(DEV) for t in orc.make_blast_inputs(N, 512, 768, 4, 128, torch.float16, seed=seed))
        x, q8 = x.reshape(N, 512), (*bq.quantize_blast_factors(U, Vt, 8), S)
        w1, w2, half = U[:, :64, :].contiguous(), Vt[:, :, :64].contiguous(), (U[:2].contiguous(), Vt, S[:2].contiguous())
        calls = [lambda: bk.blast_torch_layout(x, U, Vt, S), lambda: bq.blast_wq(x, *q8, 8), lambda: mk.monarch_torch_layout(x, w1, w2),
                 lambda: bk.blast_output_blocks(x, *half), lambda: bk.blast_multi_torch_layout(x, [(U, Vt, S)] * 2)[1]]
        return [(c, c()) for c in calls]

    sets = [layer(1, 4), layer(2, 40), layer(3, 16)]
    torch.cuda.synchronize()

    def many(calls):
        for _ in range(60):
            for call, want in calls:
                assert torch.equal(call(), want)

    _together(*(lambda s=s: many(s) for s in sets))


def test_host_calls_of_two_threads_on_one_stream():
    """The slots of the staging ring belong to one call each."""
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    sets = []
    for seed in (1, 2):
        x, U, Vt, S = (t.to(DEV) for t in orc.make_blast_inputs(4, 512, 768, 4, 128, torch.float16, seed=seed))
        factors = (*bq.quantize_blast_factors(U, Vt, 8), S)
        want = bq.blast_wq_host(x.reshape(4, 512).cpu().pin_memory(), *factors, 8)
        bq.host_flush()
        torch.cuda.synchronize()
        sets.append((x.reshape(4, 512).cpu().pin_memory(), factors, want.clone()))

    def many(x, factors, want):
        outs = [bq.blast_wq_host(x, *factors, 8) for _ in range(40)]
        bq.host_flush()
        torch.cuda.synchronize()
        for out in outs:
            assert torch.equal(out, want)

    _together(*(lambda s=s: many(*s) for s in sets))


def test_two_threads_share_the_coupling_factors(monkeypatch):
    """Room for the expanded factors of one layer: each thread's call drops those of the other."""
    import mem_efficient_blr_b200.blast_kernels as bk
    from mem_efficient_blr_b200 import ops
    sets = []
    for seed in (1, 2):
        x, U, Vt, S = (t.to(DEV) for t in orc.make_blast_inputs(260, 64, 96, 4, 32, torch.float16, seed=seed))
        sets.append((x.reshape(260, 64), U, Vt, S, bk.blast_torch_layout(x.reshape(260, 64), U, Vt, S)))
    ops.clear_coupling_cache()
    monkeypatch.setattr(ops, "coupling_cache_bytes", 32 * 16 * 4 * 4 * 2)
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)

    def many(x, U, Vt, S, want):
        for _ in range(2000):
            got = bk.blast_torch_layout(x, U, Vt, S)
        assert torch.equal(got, want)

    try:
        _together(*(lambda s=s: many(*s) for s in sets * 2))
    finally:
        sys.setswitchinterval(interval)
    assert len(ops._coupling) == 1 and ops._coupling_held == ops.coupling_cache_bytes
    ops.clear_coupling_cache()
