"""Reconstruction from two threads with different numbers of components: neither lowers the other's
shared-memory limit between raising it and launching."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbins", [64, 63])  # 16-byte rows, single floats
def test_two_threads_with_different_component_counts(sfh, nbins):
    torch = pytest.importorskip("torch")
    from sfhgpu._lib import load
    L, dev, B = load(), torch.device("cuda", 0), 16
    jobs, failed = [], []
    for K in (700, 800, 900, 1024):
        g = torch.Generator(device=dev).manual_seed(K)
        basis = torch.randn((K, nbins), generator=g, device=dev) / K
        coef = torch.randn((B, K), generator=g, device=dev)
        off = torch.full((nbins,), 2.0, device=dev)
        rows = torch.arange(B, dtype=torch.int32, device=dev)
        seg = torch.tensor([[0, 0, B]], dtype=torch.int32, device=dev)
        out = torch.empty((B, nbins), device=dev)
        jobs.append((K, sfh.Context(0), coef, rows, seg, basis, off, out))
    torch.cuda.synchronize()

    def work(K, ctx, coef, rows, seg, basis, off, out):
        for _ in range(4000):
            rc = L.sfh_emu_reconstruct_groups(
                ctx.handle, coef.data_ptr(), rows.data_ptr(), seg.data_ptr(), 1, 1, basis.data_ptr(),
                off.data_ptr(), K, nbins, B, 0, out.data_ptr())
            if rc:
                failed.append((K, rc))
                return
        ctx.synchronize()
    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for K, _, coef, _, _, basis, off, out in jobs:
        ref = coef.double() @ basis.double() + off.double()
        # K products of magnitudes near 1 / K, FP32 sums
        assert np.max(np.abs(out.cpu().numpy() - ref.clamp(min=0).cpu().numpy())) < 1e-5
