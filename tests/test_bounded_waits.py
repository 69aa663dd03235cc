"""Failure detection on the device without faulting one: peers that never arrive.

``Fabric(silent_peers=True)`` maps the other ranks to blocks on this GPU that nothing writes, with a small poll limit. Every
fused collective must give up after its bounded wait, record PEER_TIMEOUT in the sticky status word and return; the context
stays usable, and after the status is cleared a one-rank fabric computes correct results on the same device."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
MBAR_TIMEOUT = 2


def _status_bits():
    from ironpangu_b200.parallel import fabric as F

    return {"PEER_TIMEOUT": F.STATUS_PEER_TIMEOUT}


def test_decode_collectives_time_out_and_report():
    from ironpangu_b200.ops import decode as K
    from ironpangu_b200.parallel.fabric import Fabric

    bits = _status_bits()
    fab = Fabric(0, 2, silent_peers=True, spin_limit=2000)
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(1, 512, generator=g, device="cuda").to(BF16)
    w = (torch.randn(256, 512, generator=g, device="cuda") * 0.05).to(BF16)
    assert fab.status() == 0
    K.gemv_allreduce(x, w, fab)                     # the peer's partial sums never come
    torch.cuda.synchronize()
    assert fab.status() & bits["PEER_TIMEOUT"]
    fab.clear_status()
    head = (torch.randn(1024, 512, generator=g, device="cuda") * 0.05).to(BF16)
    K.lm_head_argmax(x, head, fab)                  # the peer's (value, index) candidates never come
    torch.cuda.synchronize()
    assert fab.status() & bits["PEER_TIMEOUT"]
    fab.close()
    # the device is fine: a one-rank fabric computes the same GEMV correctly afterwards
    solo = Fabric(0, 1)
    y = K.gemv_allreduce(x, w, solo)
    torch.testing.assert_close(y.float(), (x.float() @ w.float().T), rtol=2e-2, atol=2e-2)
    assert solo.status() == 0
    solo.close()


def test_bulk_gemm_allreduce_times_out_and_frees_its_tensor_memory():
    from ironpangu_b200.ops.gemm import gemm, gemm_allreduce
    from ironpangu_b200.parallel.fabric import Fabric

    bits = _status_bits()
    fab = Fabric(0, 2, silent_peers=True, spin_limit=2000, data_half_bytes=8 << 20)
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(256, 256, generator=g, device="cuda").to(BF16)
    b = (torch.randn(512, 256, generator=g, device="cuda") * 0.05).to(BF16)

    class Sym:                                        # both "ranks" publish into buffers on this device
        def __init__(self):
            import ctypes as C
            self.tensor = torch.zeros(256, 512, dtype=BF16, device="cuda")
            self.other = torch.zeros(256, 512, dtype=BF16, device="cuda")
            self.peer_ptrs = (C.c_void_p * 8)(self.tensor.data_ptr(), self.other.data_ptr())

    sym = Sym()
    gemm_allreduce(a, b, fab, sym)
    torch.cuda.synchronize()
    assert fab.status() & bits["PEER_TIMEOUT"]
    fab.close()
    # tensor memory was released on the way out: a plain tcgen05 GEMM still gets its allocation and is correct
    c = gemm(a, b)
    torch.testing.assert_close(c.float(), a.float() @ b.float().T, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("M,N,K,F", [(5, 256, 512, 0), (8, 2048, 6144, 0), (130, 300, 1024, 0), (20, 512, 2048, 256)])
def test_few_row_product_whose_waits_run_out_reports(M, N, K, F):
    """A limit of no polls at all: every warp gives up at its first wait, what has been started is waited for, the result is NaN and the next product
    is right."""
    import ctypes as C

    from ironpangu_b200.ops import _lib
    from ironpangu_b200.ops.gemm import gemm

    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn(M, K, generator=g, device="cuda").to(BF16)
    b = (torch.randn(N, K, generator=g, device="cuda") * 0.05).to(BF16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    cols = F or N
    P, L, I, R, U = C.c_void_p, C.c_long, C.c_int, C.c_float, C.c_uint32
    lib = C.CDLL(_lib.load()._name)                 # a handle of its own: argument types are set here
    run = lib.ifab_gemm_rows_bf16
    run.argtypes = [P, L, P, L, P, L, I, P, L, P, I, R, I, R, R, I, I, I, I, I, U, P, P]

    def product(limit):
        out = torch.full((M, cols), 7.0, dtype=BF16, device="cuda")
        assert run(a.data_ptr(), K, b.data_ptr(), K, out.data_ptr(), cols, 0, None, 0, None, 0, 0.0, 0, 0.0, 1.0, F, 1, M, N, K, limit, status.data_ptr(),
                   torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        return out

    out = product(0)
    assert int(status) == MBAR_TIMEOUT and bool(out.isnan().all())
    status.zero_()
    out, full = product(4000000), a.float() @ b.float().T
    want = torch.nn.functional.silu(full[:, :F].to(BF16).float()) * full[:, F:].to(BF16).float() if F else full
    torch.testing.assert_close(out.float(), want, rtol=2e-2, atol=2e-2)
    assert int(status) == 0
    torch.testing.assert_close(gemm(a, b).float(), full, rtol=2e-2, atol=2e-2)
