"""Native calls from threads whose first CUDA call they are, as the threads that run backward passes make them."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _in_thread(fn):
    got = []

    def body():
        try:
            got.append(fn())
        except BaseException as e:      # (shown by the caller)
            got.append(e)

    t = threading.Thread(target=body)
    t.start()
    t.join()
    if isinstance(got[0], BaseException):
        raise got[0]
    return got[0]


@pytest.mark.parametrize("M", [8, 640])
@pytest.mark.parametrize("what", ["gemm", "flash", "decode"])
def test_first_call_of_a_thread(what, M):
    """Results come out of cached memory, so that nothing has made the device's context the thread's before."""
    from litetorch_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = (torch.randn(n, 512, device="cuda", generator=g).bfloat16() for n in (M, 1024))
    q = torch.randn(1, M, 4, 64, device="cuda", generator=g).bfloat16()
    kc = torch.randn(M, 4, 16, 64, device="cuda", generator=g).bfloat16()
    table, lens = torch.arange(M, dtype=torch.int32, device="cuda").view(M, 1), torch.full((M,), 9, dtype=torch.int32, device="cuda")
    fn = {"gemm": lambda: K.gemm(x, w), "flash": lambda: K.flash_fwd(q, q, q)[0],
          "decode": lambda: K.paged_decode(q[0], kc, kc, table, lens, 16, 1, 0.125)}[what]
    want = fn()
    torch.cuda.synchronize()
    for _ in range(3):
        keep = fn()
        torch.cuda.synchronize()
        del keep                        # its memory is what the thread gets
        got = _in_thread(fn)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
        del got
    assert K.status_fetch() == 0
