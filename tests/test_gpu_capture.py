"""Workspaces that come into being inside a stream capture: what the recorded work would have zeroed is not zero yet."""
import os
import subprocess
import sys

import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
HEAD = 1024 + (2 << 20)   # control words and accumulation area, zero between calls


@pytest.mark.parametrize("path", [1, 2])   # grid-wide kernel (barrier words), cluster kernel (arrival counters, fp32 sums)
def test_captured_workspace(path):
    import mem_efficient_blr_b200.blast_kernels as bk
    from mem_efficient_blr_b200 import _lib as L
    dev, lib = torch.device(DEV), L.load()
    x, U, Vt, S = (t.to(DEV) for t in orc.make_blast_inputs(4, 512, 768, 4, 128, torch.float16, seed=1))
    want = orc.blast(*(t.cpu() for t in (x, U, Vt, S)))[0].reshape(x.shape[:-1] + (768,))
    right = lambda y: orc.rel_fro(y.float().cpu().reshape(want.shape), want) < 1e-2
    call = lambda: bk.blast_torch_layout(x, U, Vt, S)
    st = torch.cuda.Stream()
    L.check(lib.blr_debug_decode_path(path))
    try:
        graphs = []
        for i in range(2):
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                if i == 0:   # a buffer of its own for this capture, whatever the stream had
                    old = L.workspace(dev, st.cuda_stream, HEAD)
                    ws = L.workspace(dev, st.cuda_stream, old.numel() + HEAD)
                y = call()
            graphs.append((g, y))

        def leave_anything():
            ws[:HEAD] = 0xFF
            torch.cuda.synchronize()

        leave_anything()
        g, y = graphs[1]   # the second graph, without ever running the first
        g.replay()
        torch.cuda.synchronize()
        assert right(y)
        leave_anything()
        with torch.cuda.stream(st):   # a call outside of any graph
            assert L.workspace(dev, st.cuda_stream, HEAD).data_ptr() == ws.data_ptr()
            y = call()
        torch.cuda.synchronize()
        assert right(y)
        graphs[0][0].replay()
        torch.cuda.synchronize()
        assert right(graphs[0][1])
        with torch.cuda.stream(st):
            L.workspace_status(dev)
    finally:
        L.check(lib.blr_debug_decode_path(0))


def test_captured_workspace_without_the_extension():
    """The same through ctypes, whose workspaces the Python layer keeps."""
    if os.environ.get("BLR_B200_NO_TORCH_EXT"):
        pytest.skip("this is the process without the extension")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", __file__, "-m", "gpu"], env={**os.environ, "BLR_B200_NO_TORCH_EXT": "1"},
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
