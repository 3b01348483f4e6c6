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


# the host route: fewer than 16,384 blocks; a stride or a destination that 16-byte stores cannot take.  The device's: from 16,384
# blocks on; a last CTA of 16, 240 and 256 of its 256 blocks; one block row short of, at and past a 32,768-block staging slot; several
# slots; experts that end inside a CTA
@pytest.mark.parametrize("M,K,e0,e1,offset", [(16, 32, 0, 1, 0), (16, 32, 2, 5, 0), (240, 32, 0, 1, 0), (256, 32, 0, 1, 0), (272, 32, 0, 3, 0),
                                              (2047 * 16, 32, 0, 1, 0), (2048 * 16, 32, 0, 1, 0), (2049 * 16, 32, 0, 2, 0),
                                              (512, 2048, 1, 12, 0), (17, 32, 0, 3, 0), (16, 96, 0, 2, 0), (16, 32, 0, 3, 8),
                                              (1023 * 16, 32, 0, 1, 0), (1024 * 16, 32, 0, 1, 0), (1025 * 16, 32, 0, 1, 0),
                                              (1039 * 16, 32, 0, 1, 0), (1040 * 16, 32, 0, 1, 0), (16, 32, 3, 1027, 0), (48, 96, 2, 177, 0),
                                              (1025 * 16, 32, 0, 2, 8), (4097, 128, 0, 1, 0)])
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


_OWN_CONTEXT = """
import ctypes as C, sys
import numpy as np
from q36_b200 import moe
cu = C.CDLL("libcuda.so.1")
def ok(rc): assert rc == 0, rc
ctx, cur, dst = C.c_void_p(), C.c_void_p(), C.c_uint64()
ok(cu.cuInit(0))
ok(cu.cuCtxCreate_v2(C.byref(ctx), 0, 0))
M, K, n = 512, 2048, 8                                  # eight staging slots: several threads
blocks = np.random.default_rng(0).integers(0, 256, size=(n, M, K // 32, 17), dtype=np.uint8)
want, got = np.empty(n * moe.expert_stride(M, K), np.uint8), np.empty(n * moe.expert_stride(M, K), np.uint8)
moe.check(moe.lib.q36_moe_repack_mxfp4(blocks.ctypes.data, K, M, 0, n, want.ctypes.data), "repack")
ok(cu.cuMemAlloc_v2(C.byref(dst), C.c_size_t(want.size)))
for i in range(2):
    moe.check(moe.lib.q36_moe_upload_mxfp4(blocks.ctypes.data, K, M, 0, n, dst.value), "upload")
    ok(cu.cuCtxGetCurrent(C.byref(cur)))
    assert cur.value == ctx.value                        # the caller's thread stays in its context
    ok(cu.cuMemcpyDtoH_v2(C.c_void_p(got.ctypes.data), dst, C.c_size_t(got.size)))
    assert (got == want).all()
    moe.check(moe.lib.q36_moe_upload_release(), "release")
ok(cu.cuMemsetD8_v2(dst, 0, C.c_size_t(got.size)))
prim = C.c_void_p()
ok(cu.cuDevicePrimaryCtxRetain(C.byref(prim), 0))
ok(cu.cuCtxSetCurrent(prim))                             # the memory of one context, uploaded to from another
moe.check(moe.lib.q36_moe_upload_mxfp4(blocks.ctypes.data, K, M, 0, n, dst.value), "upload")
ok(cu.cuCtxSetCurrent(ctx))
ok(cu.cuMemcpyDtoH_v2(C.c_void_p(got.ctypes.data), dst, C.c_size_t(got.size)))
assert (got == want).all()
"""


def test_upload_in_a_context_of_the_programs_own(moe):
    """A program may work in a context of its own instead of the runtime's primary one, as with a plain copy."""
    import os
    import subprocess
    import sys
    r = subprocess.run([sys.executable, "-c", _OWN_CONTEXT], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr[-2000:]


# gate/up tiles of 32 ff rows while the groups' tiles are at most the SMs (148: 9 groups x 16), 64 up to 18 groups, then 128
@pytest.mark.parametrize("k,T,se0,se1,shared", [(4, 1, 0, 32, True), (8, 1, 0, 32, True), (8, 1, 0, 32, False), (4, 2, 0, 32, True),
                                                (2, 3, 0, 32, True), (4, 3, 0, 32, True), (8, 2, 0, 32, True), (4, 4, 0, 32, True),
                                                (8, 3, 0, 32, True), (8, 16, 8, 16, False), (8, 16, 8, 24, False), (8, 40, 0, 8, True),
                                                (4, 100, 24, 32, False)])
def test_gateup_tile_heights_agree_with_the_cuda_core_path(moe, k, T, se0, se1, shared):
    import torch
    ly = moe.MoELayer(n_expert=32, k=k, se0=se0, se1=se1).random_planes(3 + k, shared=shared)
    rng = np.random.default_rng(10 * T + k)
    X = torch.from_numpy(synth.activations(rng, T)).cuda().to(torch.bfloat16)
    L = torch.from_numpy(synth.router_logits(rng, T, 32)).cuda()
    a = ly.forward(X, L, path=moe.PATH_TC, inc_shared=shared)
    ly.check_device_status()
    b = ly.forward(X, L, path=moe.PATH_GEMV, inc_shared=shared)
    # f32 sums in another order; a value of the E4M3 intermediate on a rounding boundary may fall on its other side (1e-3 of its row)
    assert float(b.abs().max()) > 0 and rel_l2(a, b) < 2e-3


def test_gateup_tile_heights_give_the_same_bits(moe):
    """A token's result does not depend on the tile height: calls of one token (9 groups: tiles of 32 ff rows), two (18: 64 rows)
    and all sixteen (128 rows) sum the same products in the same order."""
    import torch
    T = 16
    ly = moe.MoELayer(n_expert=64, k=8).random_planes(5)
    rng = np.random.default_rng(5)
    X = torch.from_numpy(synth.activations(rng, T)).cuda().to(torch.bfloat16)
    L = torch.from_numpy(synth.router_logits(rng, T, 64)).cuda()
    want = ly.forward(X, L)
    for n in (1, 2):
        got = torch.cat([ly.forward(X[t:t + n].contiguous(), L[t:t + n].contiguous()) for t in range(0, T, n)])
        ly.check_device_status()
        assert torch.equal(got, want), f"{n} token(s) per call"


# placed by the scan's cluster up to 4096 entries, by a launch of its own beyond; entries of other ranks and without an expert
@pytest.mark.parametrize("n", [1, 511, 4095, 4096, 4097, 16384, 70001])
@pytest.mark.parametrize("E,se0,se1", [(256, 0, 256), (64, 16, 48), (512, 100, 512)])
def test_dispatch_places_every_entry(moe, n, E, se0, se1):
    import torch
    rng = np.random.default_rng(n + E)
    eid = rng.integers(-1, E, size=n, dtype=np.int32)
    ecount, eoffs, elist, pos = moe.dispatch(torch.from_numpy(eid).cuda(), E, se0, se1)
    mine = (eid >= se0) & (eid < se1)
    want_count = np.bincount(eid[mine], minlength=E)
    want_list = np.flatnonzero(mine)[np.argsort(eid[mine], kind="stable")]
    want_pos = np.full(n, -1)
    want_pos[want_list] = np.arange(want_list.size)
    np.testing.assert_array_equal(ecount.cpu().numpy(), want_count)
    np.testing.assert_array_equal(eoffs.cpu().numpy(), np.concatenate([[0], np.cumsum(want_count)]))
    np.testing.assert_array_equal(elist.cpu().numpy()[:want_list.size], want_list)
    np.testing.assert_array_equal(pos.cpu().numpy(), want_pos)


# cluster front end up to 512 tokens at k = 8, 680 at k = 6, 768 at k <= 5, two launches beyond; the decode cluster up to 16
@pytest.mark.parametrize("E,k,T", [(E, k, T) for E, k in ((256, 8), (128, 6), (64, 1), (32, 8))
                                   for T in (16, 17, 63, 64, 65, 511, 512, 513, 1025)] +
                         [(128, 6, 680), (128, 6, 681)] + [(E, k, T) for E, k in ((256, 1), (64, 2), (32, 4), (128, 5)) for T in (768, 769)])
def test_front_end_of_any_batch(moe, oracle, E, k, T):
    import torch
    rng = np.random.default_rng(T + E)
    L = synth.router_logits(rng, T, E, zipf=T % 2 == 1)
    L[T // 2, : E // 2] = 0.25                               # ties: the lower id wins
    ly = moe.MoELayer(n_expert=E, k=k).random_planes(E)
    X = torch.from_numpy(synth.activations(rng, T)).cuda().to(torch.bfloat16)
    lt = torch.from_numpy(L).cuda()
    out, idx, wt = ly.forward(X, lt, want_routing=True)
    ly.check_device_status()
    sidx, swt = moe.router_topk(lt, E, k)                    # the router entry on its own
    assert torch.equal(idx, sidx) and torch.equal(wt, swt)
    widx, _ = oracle.router_topk(L, k, n_expert=E)
    np.testing.assert_array_equal(idx.cpu().numpy(), widx)
    want = ly.forward(X, lt, path=moe.PATH_GEMV)
    assert rel_l2(out, want) < 2e-3                          # as above


def test_router_rows_without_a_largest_value(moe):
    """NaN, infinities and the lowest values: every route must choose what the router entry chooses."""
    import torch
    E, k = 64, 4
    low = torch.finfo(torch.float32).min
    for T in (8, 40, 600):
        g = torch.Generator(device="cuda")
        g.manual_seed(T)
        L = torch.randn((T, E + 1), device="cuda", generator=g)
        L[0, :E] = float("-inf")
        L[1, :E] = low
        L[2, 3] = float("nan")
        L[3, 5:] = float("-inf")
        L[4, 7] = float("inf")
        L[5, 2:] = low                                       # two experts to choose from, four wanted
        ly = moe.MoELayer(n_expert=E, k=k).random_planes(1)
        X = torch.randn((T, D), device="cuda", generator=g)
        _, idx, wt = ly.forward(X, L, want_routing=True)
        ly.check_device_status()
        sidx, swt = moe.router_topk(L, E, k)
        assert torch.equal(idx, sidx) and torch.equal(wt.isnan(), swt.isnan())
        assert torch.equal(wt.nan_to_num(), swt.nan_to_num())
        assert int(idx.min()) >= 0 and int(idx.max()) < E


def _choices(row, k):
    """The selection rule in plain words: largest first, the lower id among equals, what is NaN or at most -1e30 never; expert 0 fills
    the slots that stay empty."""
    ids = [e for e in range(len(row)) if row[e] > -1e30]
    ids.sort(key=lambda e: (-float(row[e]), e))
    return (ids + [0] * k)[:k]


@pytest.mark.parametrize("E,k", [(32, 8), (64, 4), (128, 1), (256, 8), (256, 3)])
@pytest.mark.parametrize("T", [12, 40, 600])                 # the decode cluster, the batch cluster, the two launches
def test_router_choices_by_definition(moe, E, k, T):
    import torch
    rng = np.random.default_rng(E + k)
    L = rng.standard_normal((T, E + 1), dtype=np.float32)
    low = np.finfo(np.float32).min
    L[0, :E] = -np.inf
    L[1, :E] = low
    L[2, 3] = np.nan
    L[3, 5:E] = -np.inf
    L[4, 7] = np.inf
    L[5, 2:E] = low
    L[6, :E] = 0.5                                           # every value ties
    L[7, :E] = np.where(np.arange(E) % 2, 0.0, -0.0)         # ... and these do
    L[8, E // 4:] = 3.0                                      # more than a warp's worth tie for the first place
    L[9, :E] = np.float32(-1e30)
    L[10, :E] = np.nan
    L[11, :E] = np.sort(L[11, :E])
    lt = torch.from_numpy(L).cuda()
    ly = moe.MoELayer(n_expert=E, k=k).random_planes(1)
    X = torch.from_numpy(synth.activations(rng, T)).cuda()
    _, idx, wt = ly.forward(X, lt, want_routing=True)
    ly.check_device_status()
    sidx, swt = moe.router_topk(lt, E, k)
    want = np.array([_choices(L[t, :E], k) for t in range(T)])
    for i, w in ((idx, wt), (sidx, swt)):
        np.testing.assert_array_equal(i.cpu().numpy(), want)
        w = w.cpu().numpy()
        for t in range(T):
            v = L[t, :E].astype(np.float64)
            if not np.isfinite(v[want[t]]).all() or not (v > -1e30).any() or np.isnan(v).any():
                continue
            e = np.where(np.arange(k) < (v > -1e30).sum(), np.exp(v[want[t]] - v.max()), 0.0)      # an empty slot weighs nothing
            # exponentials and two quotients in f32: a few ulps each
            np.testing.assert_allclose(w[t], e / e.sum(), rtol=3e-6, atol=1e-12)


# the logits kernels: rows in registers (1, 2, 4, 8, 16 tokens), then 32-, 64- and 128-token tiles with K split 8 or 4 ways, and from
# 2.2 tiles per SM on (326 tiles of 128 x 64) unsplit
@pytest.mark.parametrize("T,n_rows", [(1, 33), (2, 257), (3, 65), (5, 257), (9, 129), (16, 257), (17, 257), (33, 33), (128, 257), (129, 129),
                                      (1000, 257), (1025, 257), (4097, 33), (10368, 257), (10369, 257), (20000, 257), (41601, 33)])
def test_router_logits_at_the_changes_of_tile(moe, T, n_rows):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(T)
    h = torch.randn((T, D), device="cuda", generator=g)
    w = 1 + 0.1 * torch.randn(D, device="cuda", generator=g)
    router = torch.randn((n_rows, D), device="cuda", generator=g) / D ** 0.5
    x, logits = moe.pre_norm_router(h, None, w, router, gate_row=n_rows - 1)
    want = x.double() @ router.double().T
    # sums of 2048 f32 products whose partial sums stay below a few units: far below 2048 ulps of the largest
    assert float((logits.double() - want).abs().max()) < 2e-5 * float(want.abs().max())


def test_decode_rows_with_one_eligible_expert(moe):
    """Rows whose other logits are masked out fill their remaining slots with expert 0 at weight 0: 16 tokens then have 112
    entries of that expert, more than one 16-row token tile."""
    import torch
    E, k, T = 32, 8, 16
    L = torch.full((T, E + 1), float("-inf"), device="cuda")
    L[torch.arange(T), 1 + torch.arange(T)] = 1.0
    L[:, E] = 0.5
    ly = moe.MoELayer(n_expert=E, k=k).random_planes(2)
    X = torch.from_numpy(synth.activations(np.random.default_rng(2), T)).cuda().to(torch.bfloat16)
    out = ly.forward(X, L)
    ly.check_device_status()
    want = ly.forward(X, L, path=moe.PATH_GEMV)
    assert bool(torch.isfinite(want).all()) and rel_l2(out, want) < 2e-3


# hidden 4096 is beyond the decode kernel: the grouped-GEMM launches follow the front end at every batch, and need its plan in their
# own token tiles; with one eligible expert per row 56 of the 64 rows fall to expert 0
@pytest.mark.parametrize("T,masked", [(1, False), (8, False), (8, True), (9, False)])
def test_decode_batches_of_a_layer_the_decode_kernel_does_not_take(moe, T, masked):
    import torch
    E, k, D4 = 32, 8, 4096
    assert not moe.lib.q36_moe_one_launch_fits(T * (k + 1), E, D4, FF)
    ly = moe.MoELayer(n_expert=E, k=k, D=D4).random_planes(4)
    rng = np.random.default_rng(T)
    X = torch.from_numpy(synth.activations(rng, T, D4)).cuda().to(torch.bfloat16)
    L = torch.from_numpy(synth.router_logits(rng, T, E)).cuda()
    if masked:
        L[:, :E] = float("-inf")
        L[torch.arange(T), 1 + torch.arange(T)] = 1.0
    out = ly.forward(X, L)
    ly.check_device_status()
    want = ly.forward(X, L, path=moe.PATH_GEMV)
    # f32 sums in another order; E4M3 values of the intermediate on a rounding boundary (1e-3 of a row)
    assert bool(torch.isfinite(want).all()) and float(want.abs().max()) > 0 and rel_l2(out, want) < 2e-3
