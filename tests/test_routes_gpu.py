"""The rules that choose a kernel variant by size or alignment, at the sizes where they change over: each variant against the
general one, or against the oracle, through the C ABI."""
import threading

import numpy as np
import pytest

from q36_b200 import synth

pytestmark = pytest.mark.gpu

D, FF = synth.D_MODEL, synth.EXPERT_FF


def rel_l2(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm())


# one block short of, at and past a 256-block CTA and a 32,768-block staging slot; several slots; a stride or a destination
# that 16-byte stores cannot take (the host route)
@pytest.mark.parametrize("M,K,e0,e1,offset", [(16, 32, 0, 1, 0), (16, 32, 2, 5, 0), (240, 32, 0, 1, 0), (256, 32, 0, 1, 0), (272, 32, 0, 3, 0),
                                              (2047 * 16, 32, 0, 1, 0), (2048 * 16, 32, 0, 1, 0), (2049 * 16, 32, 0, 2, 0),
                                              (512, 2048, 1, 12, 0), (17, 32, 0, 3, 0), (16, 96, 0, 2, 0), (16, 32, 0, 3, 8)])
def test_upload_equals_the_host_repack(moe, M, K, e0, e1, offset):
    import torch
    rng = np.random.default_rng(M + K)
    blocks = rng.integers(0, 256, size=(e1, M, K // 32, 17), dtype=np.uint8)
    n = (e1 - e0) * moe.expert_stride(M, K)
    want = np.empty(n, np.uint8)
    moe.check(moe.lib.q36_moe_repack_mxfp4(blocks.ctypes.data, K, M, e0, e1, want.ctypes.data), "repack")
    buf = torch.full((n + 32,), 0xA5, dtype=torch.uint8, device="cuda")
    moe.check(moe.lib.q36_moe_upload_mxfp4(blocks.ctypes.data, K, M, e0, e1, buf.data_ptr() + offset), "upload")
    got = buf.cpu().numpy()
    np.testing.assert_array_equal(got[offset:offset + n], want)
    assert (got[:offset] == 0xA5).all() and (got[offset + n:] == 0xA5).all()      # nothing around it is touched
    moe.check(moe.lib.q36_moe_upload_release(), "release")                        # (the next upload pins its staging anew)


def test_uploads_from_several_threads_do_not_disturb_each_other(moe):
    rng = np.random.default_rng(1)
    jobs = [rng.integers(0, 256, size=(3, 1024, 64, 17), dtype=np.uint8) for _ in range(4)]
    got = [None] * len(jobs)

    def work(i):
        got[i] = moe.upload_mxfp4(jobs[i], 2048, 1024, 0, 3)
    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for b, g in zip(jobs, got):
        want = np.empty(g.numel(), np.uint8)
        moe.check(moe.lib.q36_moe_repack_mxfp4(b.ctypes.data, 2048, 1024, 0, 3, want.ctypes.data), "repack")
        np.testing.assert_array_equal(g.cpu().numpy(), want)
