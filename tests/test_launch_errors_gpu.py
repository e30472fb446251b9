"""A launch that the runtime refuses (on the host: the diagnostics build gives it a block of no threads) is reported by the
call it belongs to, with its CUDA error, and is nothing to the next call on the thread."""
import pytest
import torch

from oracle import retention_oracle as orc

pytestmark = pytest.mark.gpu
INVALID_CONFIGURATION = 9                 # cudaErrorInvalidConfiguration


# (B, T, H, dk, dv, dtype): walks whole; in T-segments (state pass, scan, walk); dv in two halves; fp32 chunks in segments
@pytest.mark.parametrize("B,T,H,dk,dv,dtype,launches", [
    (2, 100, 2, 64, 64, torch.bfloat16, 1), (1, 4096, 2, 128, 128, torch.bfloat16, 3), (1, 200, 2, 128, 256, torch.bfloat16, 1),
    (1, 512, 2, 64, 64, torch.float32, 3)])
def test_a_refused_launch_is_its_own_calls_error(B, T, H, dk, dv, dtype, launches):
    import flash_pop_b200 as fp
    from flash_pop_b200 import _lib
    decays = tuple(orc.head_decays(H, (5, 12)))
    r = lambda d: (torch.randn(B, T, H, d, device="cuda") * 0.1).to(dtype).requires_grad_(True)
    q, k, v = r(dk), r(dk), r(dv)
    forward = lambda: fp.fused_chunk_retention(q, k, v, None, decays)[0]
    with _lib.diagnostics_build() as diag:
        try:
            want = forward()
            grads = torch.autograd.grad(want, [q, k, v], want.detach(), retain_graph=True)

            def refused(call, n):
                diag.fpb_debug_refuse_launch(n)
                with pytest.raises(RuntimeError, match=r"cudaError %d\]" % INVALID_CONFIGURATION):
                    call()
                diag.fpb_debug_refuse_launch(-1)
                assert torch.equal(forward(), want)
                got = torch.autograd.grad(want, [q, k, v], want.detach(), retain_graph=True)
                assert all(torch.equal(a, b) for a, b in zip(got, grads))

            for n in range(launches):
                refused(forward, n)
            backward = lambda: torch.autograd.grad(want, [q, k, v], want.detach(), retain_graph=True)
            for n in range(launches if dtype == torch.float32 else launches + 1):
                refused(backward, n)
        finally:
            diag.fpb_debug_refuse_launch(-1)
    torch.cuda.synchronize()
    _lib.device_status()
