"""The workspace of a stream under several threads: growth by one thread beside calls of another."""
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
