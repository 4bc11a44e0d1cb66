"""Stage-wise parity of the CUDA kernels against the CPU oracle, through the C ABI.

Every stage is fed the same inputs as the oracle; integer outputs (labels,
counts, permutations, bitmaps, row counts) and order-defined sums must match
bit for bit, tensor-core products within a stated tolerance.
"""
import math

import pytest
import torch

from oracle import t2t_oracle as O

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
DEV = "cuda"


def _st():
    return torch.cuda.current_stream().cuda_stream


def _ok(code):
    assert code == 0, f"C ABI returned {code}"


def test_gather4_selftest(lib):
    """Four-row TMA gathers fill a 128-byte-swizzled tile exactly as the manual
    16-byte copies of the other kernels do."""
    g = torch.Generator().manual_seed(11)
    rows = 1000
    src = torch.randn(rows, 128, generator=g).to(BF)
    gidx = torch.randint(0, rows, (128,), generator=g, dtype=torch.int32)
    gidx[5] = gidx[4]                      # repeated rows are allowed
    gidx[127] = rows - 1
    out = torch.zeros(32768, dtype=torch.uint8, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    srcd, gd = src.to(DEV), gidx.to(DEV)
    _ok(lib.t2t_gather4_selftest(srcd.data_ptr(), rows, gd.data_ptr(), out.data_ptr(), status.data_ptr(), _st()))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    got = out.cpu().view(torch.int16).view(2, 128, 8, 8)          # [block][row][stored chunk][8 values]
    want = src[gidx.long()].view(torch.int16).view(128, 2, 8, 8).permute(1, 0, 2, 3)   # [block][row][chunk][8]
    r = torch.arange(128)[:, None]
    c = torch.arange(8)[None, :]
    stored = (c ^ (r & 7)).long()                                   # chunk c of row r lives at chunk c ^ (r & 7)
    unsw = torch.gather(got, 2, stored[None, :, :, None].expand(2, 128, 8, 8))
    assert torch.equal(unsw, want)


def test_bounded_wait_gives_up_cleanly(lib):
    """A wait that can never complete ends by its spin limit, raises the abort
    flag for the other warps, reports through the status word, and the context
    stays usable."""
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.full((2,), -1, dtype=torch.int32, device=DEV)
    _ok(lib.t2t_wait_timeout_selftest(status.data_ptr(), out.data_ptr(), _st()))
    torch.cuda.synchronize()
    assert int(status.item()) == 1 and out.tolist() == [0, 0]
    assert float((torch.ones(4, device=DEV) * 2).sum()) == 8.0      # the device still works


def _softmax_give_up(lib, commits, handed):
    out = torch.full((128, 128), -1.0, dtype=BF, device=DEV)
    lse = torch.full((128,), -1.0, device=DEV)
    left = torch.zeros(8, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    _ok(lib.t2t_softmax_give_up_selftest(commits, handed, out.data_ptr(), lse.data_ptr(), left.data_ptr(),
                                         status.data_ptr(), _st()))
    torch.cuda.synchronize()
    assert left.tolist() == [1] * 8
    return int(status.item()), out.float().cpu(), lse.cpu()


@pytest.mark.parametrize("commits, handed", [(0, 0), (0, 0xffffffff), (2, 0), (2, 1), (2, 0x55555555), (2, 0xffff0000),
                                             (2, 0xfffffffe)])
def test_softmax_warps_give_up_as_warps(lib, commits, handed):
    """No scores at all, or those of tile 1 alone, with the maximum behind tile 0 there for no lane of a warp, one, half of
    them, all but one: the lanes that have it must not go on to warp-collective instructions without the others."""
    status, out, lse = _softmax_give_up(lib, commits, handed)
    assert status == 1 and bool((out == -1).all()) and bool((lse == -1).all())
    assert float((torch.ones(4, device=DEV) * 2).sum()) == 8.0      # the device still works


@pytest.mark.parametrize("commits, handed", [(1, 0), (2, 0xffffffff), (3, 0), (7, 0), (19, 0), (1 | 16, 0)])
def test_softmax_warps_do_not_wait_for_a_warp_that_gave_up(lib, commits, handed):
    """One of the two warps of a row leaves at a wait that runs out (the scores of tile 1, of tile 0, the weighted sum that
    a rising maximum rescales) when the other has finished its tile and comes to where their sums are joined; or both are
    through and the last weighted sum never comes."""
    status, out, lse = _softmax_give_up(lib, commits, handed)
    assert status == 1 and bool((out == -1).all()) and bool((lse == -1).all())
    assert float((torch.ones(4, device=DEV) * 2).sum()) == 8.0      # the device still works


@pytest.mark.parametrize("commits", [15, 31])
def test_softmax_warps_join_their_sums_when_nothing_is_missing(lib, commits):
    """256 equal scores: weights of one that sum to 256, half from either warp.  Scores of 1000 in the odd rows of tile 1:
    tile 0 and the O it left weigh 2^-127.5, the second warp's 128 keys are all there is."""
    status, out, lse = _softmax_give_up(lib, commits, 0)
    odd = (torch.arange(128) % 2 == 1) & (commits == 31)
    assert status == 0 and torch.equal(out, torch.where(odd, 0.0, 1.0)[:, None].expand(128, 128))
    want = torch.where(odd, 1000.0 / math.sqrt(128.0) + math.log(128.0), math.log(256.0))
    assert (lse - want).abs().max() < 1e-4


@pytest.mark.parametrize("stuck", [-1, 0, 1, 5, 7])
def test_selection_groups_outlive_a_group_that_gave_up(lib, stuck):
    """One column group's wait runs out while the others are at work: their warps see the abort flag at different chunks and
    must still meet at their groups' barriers until the last of them is through."""
    left = torch.zeros(32, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    for _ in range(8):
        left.zero_()
        _ok(lib.t2t_select_give_up_selftest(stuck, left.data_ptr(), status.data_ptr(), _st()))
        torch.cuda.synchronize()
        assert left[:4].tolist() == [1 + stuck if stuck >= 0 else 33] * 4
        assert 1 <= int(left.min()) and int(left.max()) <= 33
        assert stuck >= 0 or left.tolist() == [33] * 32
    assert int(status.item()) == (1 if stuck >= 0 else 0)
    assert float((torch.ones(4, device=DEV) * 2).sum()) == 8.0      # the device still works


def test_umma_selftest(lib):
    g = torch.Generator().manual_seed(7)
    A = (torch.randn(128, 128, generator=g) * 0.5).to(BF)
    B = (torch.randn(128, 128, generator=g) * 0.5).to(BF)
    V = torch.randn(128, 128, generator=g).to(BF)
    S = torch.zeros(128, 128, device=DEV)
    Oo = torch.zeros(128, 128, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    Ad, Bd, Vd = A.to(DEV), B.to(DEV), V.to(DEV)
    _ok(lib.t2t_umma_selftest(Ad.data_ptr(), Bd.data_ptr(), Vd.data_ptr(), S.data_ptr(), Oo.data_ptr(),
                              status.data_ptr(), _st()))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    S_ref = A.float() @ B.float().T
    assert torch.allclose(S.cpu(), S_ref, atol=1e-3, rtol=1e-4), (S.cpu() - S_ref).abs().max()
    # accumulation error of the tensor core against the real sum, relative to sum |a||b|: the assignment
    # and selection kernels assume it is below 2^-16
    S64 = A.double() @ B.double().T
    mag = A.double().abs() @ B.double().abs().T
    kappa = float(((S.cpu().double() - S64).abs() / mag).max())
    print(f"tensor-core accumulation error: {kappa:.3e} of sum|a||b| (2^{math.log2(kappa):.1f})")
    assert kappa < 2.0 ** -18
    P = (S.cpu() * 0.0625).to(BF).float()
    O_ref = P @ V.float()
    assert torch.allclose(Oo.cpu(), O_ref, atol=2e-3, rtol=1e-4), (Oo.cpu() - O_ref).abs().max()


def test_project(lib, small_case):
    c = small_case
    x, U = c["q"].to(DEV), c["state"]["Uq"].to(DEV)
    out = torch.empty(c["H"], c["N"], 32, dtype=BF, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    _ok(lib.t2t_project(x.data_ptr(), U.data_ptr(), out.data_ptr(), c["H"], c["N"], status.data_ptr(), _st()))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    exact = torch.bmm(c["q"].float(), c["state"]["Uq"].float())
    got = out.cpu().float()
    # one bf16 rounding of an fp32-accumulated product: at most one ulp from the exact value's rounding
    tol = exact.abs() * 2.0 ** -7 + 1e-3
    assert bool(((got - exact).abs() <= tol).all())
    assert (got == exact.to(BF).float()).float().mean() > 0.98


def _assign(lib, x, cen, pin_begin=-1, pin_label=0):
    """Tensor-core assignment; also checks it against the all-exact kernel."""
    H, N, _ = x.shape
    lab = torch.empty(H, N, dtype=torch.int32, device=DEV)
    lab_exact = torch.empty_like(lab)
    ws = torch.empty(lib.t2t_assign_ws_bytes(H, N), dtype=torch.uint8, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    _ok(lib.t2t_assign(x.data_ptr(), cen.data_ptr(), lab.data_ptr(), H, N, cen.shape[1], pin_begin, pin_label,
                       ws.data_ptr(), ws.numel(), status.data_ptr(), _st()))
    _ok(lib.t2t_assign_exact(x.data_ptr(), cen.data_ptr(), lab_exact.data_ptr(), H, N, cen.shape[1], pin_begin,
                             pin_label, _st()))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert torch.equal(lab, lab_exact)
    _assign.requeued = int(ws[:4].view(torch.int32).item())
    return lab


def test_assign_tensor_core_path_equals_exact_path_at_scale(lib):
    """480p-sized random problem: the tensor-core labels must equal the all-exact
    labels, with only a small share of rows sent to the exact re-evaluation."""
    from token2tile_b200.synth import GRIDS, locality_mixture
    H, N = 4, 32760
    q, k, _ = locality_mixture(H, GRIDS["480p"])
    g = torch.Generator().manual_seed(5)
    U = (torch.randn(H, 128, 32, generator=g) * 0.1).to(BF)
    x = torch.bmm(k.float(), U.float()).to(BF).to(DEV)
    for Cn in (2048, 256):
        idx = torch.randperm(N, generator=g)[:Cn].sort().values
        cen = x[:, idx.to(DEV), :].contiguous()
        _assign(lib, x, cen)
        assert _assign.requeued < 0.05 * H * N, _assign.requeued


def test_assign_bit_exact(lib, small_case):
    c = small_case
    QU = O.project(c["q"], c["state"]["Uq"], BF)
    KU = O.project(c["k"], c["state"]["Uk"], BF)
    for x, cen, pin in ((QU, c["state"]["cq"], 0), (KU, c["state"]["ck"], 0), (KU, c["state"]["ck"], 100)):
        want = O.assign(x, cen, pin)
        got = _assign(lib, x.to(DEV), cen.to(DEV), c["N"] - pin if pin else -1, cen.shape[1] - 1)
        assert torch.equal(got.cpu(), want)


def test_assign_ties_go_to_lowest_index(lib):
    H, N, Cn = 1, 2048, 64
    g = torch.Generator().manual_seed(3)
    x = torch.randint(-3, 4, (H, N, 32), generator=g).to(BF)
    cen = torch.randint(-2, 3, (H, Cn, 32), generator=g).to(BF)
    cen[:, 10] = cen[:, 3]                      # duplicated centroids tie everywhere
    cen[:, 40] = cen[:, 3]
    want = O.assign(x, cen)
    got = _assign(lib, x.to(DEV), cen.to(DEV))
    assert torch.equal(got.cpu(), want)
    assert not bool(((want == 10) | (want == 40)).any())


def test_centroid_update_bit_exact(lib, small_case):
    c = small_case
    H, N = c["H"], c["N"]
    KU = O.project(c["k"], c["state"]["Uk"], BF)
    old = c["state"]["ck"]
    lab = O.assign(KU, old)
    lab[:, :] = torch.where(lab == 5, torch.full_like(lab, 6), lab)      # cluster 5 empty: keeps its centroid
    want_c, want_n = O.fixed_point_mean(KU, lab, old, BF)
    ws = torch.empty(lib.t2t_centroid_update_ws_bytes(H, N, 2048), dtype=torch.uint8, device=DEV)
    newc = torch.empty(H, 2048, 32, dtype=BF, device=DEV)
    counts = torch.empty(H, 2048, dtype=torch.int32, device=DEV)
    KUd, labd, oldd = KU.to(DEV), lab.to(DEV), old.to(DEV)      # keep the device copies alive
    _ok(lib.t2t_centroid_update(KUd.data_ptr(), labd.data_ptr(), oldd.data_ptr(),
                                newc.data_ptr(), counts.data_ptr(), H, N, 2048, ws.data_ptr(), ws.numel(), _st()))
    torch.cuda.synchronize()
    assert torch.equal(counts.cpu(), want_n)
    assert torch.equal(newc.cpu().view(torch.int16), want_c.view(torch.int16))


def _kmm(lib, QU, KU, V, cq0, ck0, CQ, pin_tail=0):
    H, N, _ = QU.shape
    C = 2048
    i32 = torch.int32
    e = lambda *s, dtype: torch.empty(*s, dtype=dtype, device=DEV)
    out = dict(qlab=e(H, N, dtype=i32), cq2=e(H, CQ, 32, dtype=BF), klab=e(H, N, dtype=i32),
               ck2=e(H, C, 32, dtype=torch.float32), ck16=e(H, C, 32, dtype=BF), cks16=e(H, C, 32, dtype=BF),
               qcounts=e(H, CQ, dtype=i32), qperm=e(H, N, dtype=i32), kcounts=e(H, C, dtype=i32),
               kperm=e(H, N, dtype=i32), V_sorted=e(H, N, 128, dtype=BF), sumv=e(H, C, 128, dtype=BF),
               lam=e(H, dtype=torch.float32))
    ws = torch.empty(lib.t2t_kmeans_maintain_ws_bytes(H, N, CQ, C), dtype=torch.uint8, device=DEV)
    dev = [t.to(DEV) for t in (QU, KU, V, cq0, ck0)]
    order = ["qlab", "cq2", "klab", "ck2", "ck16", "cks16", "qcounts", "qperm", "kcounts", "kperm", "V_sorted",
             "sumv", "lam"]
    _ok(lib.t2t_kmeans_maintain(*[t.data_ptr() for t in dev], *[out[k].data_ptr() for k in order],
                                1.0 / math.sqrt(128.0), H, N, CQ, C, pin_tail, ws.data_ptr(), ws.numel(), 0, _st()))
    torch.cuda.synchronize()
    return {k: t.cpu() for k, t in out.items()}


@pytest.mark.parametrize("pin_tail", [0, 77])
def test_kmeans_maintain_bit_exact(lib, small_case, pin_tail):
    c = small_case
    QU = O.project(c["q"], c["state"]["Uq"], BF)
    KU = O.project(c["k"], c["state"]["Uk"], BF)
    want = O.kmeans_maintain(QU, KU, c["v"], c["state"]["cq"], c["state"]["ck"], pin_tail, BF)
    got = _kmm(lib, QU, KU, c["v"], c["state"]["cq"], c["state"]["ck"], c["CQ"], pin_tail)
    for name in ("qlab", "klab", "qcounts", "kcounts", "qperm", "kperm"):
        assert torch.equal(got[name], want[name]), name
    assert torch.equal(got["cq2"].view(torch.int16), want["cq2"].view(torch.int16))
    assert torch.equal(got["ck2"], want["ck2"])
    assert torch.equal(got["ck16"].view(torch.int16), want["ck2"].to(BF).view(torch.int16))
    scale = 1.0 / math.sqrt(128.0)
    assert torch.equal(got["cks16"].view(torch.int16), (want["ck2"] * scale).to(BF).view(torch.int16))
    assert torch.equal(got["V_sorted"].view(torch.int16), want["V_sorted"].view(torch.int16))
    assert torch.equal(got["lam"], want["lam"])
    assert torch.equal(got["sumv"].view(torch.int16), want["sumv"].view(torch.int16))


def test_vstats_gather_and_gather_rows(lib, small_case):
    c = small_case
    H, N = c["H"], c["N"]
    KU = O.project(c["k"], c["state"]["Uk"], BF)
    klab = O.assign(KU, c["state"]["ck"])
    kcounts, kperm = O.stable_group(klab, 2048)
    v2 = (c["v"].float() * 1.5 + 0.25).to(BF)
    want_vs, want_sumv, want_lam, _ = O.vstats(v2, kperm, kcounts, BF)
    vs = torch.empty(H, N, 128, dtype=BF, device=DEV)
    sumv = torch.empty(H, 2048, 128, dtype=BF, device=DEV)
    lam = torch.empty(H, dtype=torch.float32, device=DEV)
    ws = torch.empty(lib.t2t_vstats_gather_ws_bytes(H, 2048), dtype=torch.uint8, device=DEV)
    v2d, kpermd, kcountsd, kd = v2.to(DEV), kperm.to(DEV), kcounts.to(DEV), c["k"].to(DEV)
    _ok(lib.t2t_vstats_gather(v2d.data_ptr(), kpermd.data_ptr(), kcountsd.data_ptr(),
                              vs.data_ptr(), sumv.data_ptr(), lam.data_ptr(), H, N, 2048, ws.data_ptr(),
                              ws.numel(), _st()))
    torch.cuda.synchronize()
    assert torch.equal(vs.cpu().view(torch.int16), want_vs.view(torch.int16))
    assert torch.equal(sumv.cpu().view(torch.int16), want_sumv.view(torch.int16))
    assert torch.equal(lam.cpu(), want_lam)
    kp = torch.empty(H, N, 128, dtype=BF, device=DEV)
    _ok(lib.t2t_gather_rows(kd.data_ptr(), kpermd.data_ptr(), kp.data_ptr(), H, N, _st()))
    torch.cuda.synchronize()
    want_kp = torch.gather(c["k"], 1, kperm.long()[..., None].expand(H, N, 128))
    assert torch.equal(kp.cpu().view(torch.int16), want_kp.view(torch.int16))


def _select(lib, QU, cks, kcounts, qperm, qcounts, ns, pin_tail=0):
    H, N, _ = QU.shape
    CQ = qcounts.shape[1]
    unip = torch.empty(H, CQ, 64, dtype=torch.int32, device=DEV)
    rowcnt = torch.full((H, N), -7, dtype=torch.int32, device=DEV)
    unip_x, rowcnt_x = torch.empty_like(unip), torch.empty_like(rowcnt)
    ns_t = torch.tensor(ns, dtype=torch.int32, device=DEV)
    ws = torch.empty(lib.t2t_score_select_union_ws_bytes(H, N), dtype=torch.uint8, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    dev = [t.to(DEV) for t in (QU, cks, kcounts, qperm, qcounts)]
    _ok(lib.t2t_score_select_union(*[t.data_ptr() for t in dev], ns_t.data_ptr(), unip.data_ptr(),
                                   rowcnt.data_ptr(), H, N, CQ, pin_tail, ws.data_ptr(), ws.numel(),
                                   status.data_ptr(), _st()))
    _ok(lib.t2t_score_select_union_exact(*[t.data_ptr() for t in dev], ns_t.data_ptr(), unip_x.data_ptr(),
                                         rowcnt_x.data_ptr(), H, N, CQ, pin_tail, _st()))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    # the tensor-core path and the all-exact path must agree bit for bit
    assert torch.equal(rowcnt, rowcnt_x)
    assert torch.equal(unip, unip_x)
    q = ws.view(torch.int32)[: H * (2 * N + 1)].view(H, 2 * N + 1)[:, 0]      # per head: count, then the queue
    _select.requeued = int(q.sum().item())
    return unip.cpu(), rowcnt.cpu()


def test_select_tensor_core_path_equals_exact_path_at_scale(lib):
    """480p-sized problem through real clustering: both selection paths must agree
    and only a small share of rows may need the exact re-evaluation."""
    from token2tile_b200.synth import GRIDS, locality_mixture
    H, N, CQ = 2, 32760, 256
    q, k, v = locality_mixture(H, GRIDS["480p"])
    g = torch.Generator().manual_seed(9)
    Uq = (torch.randn(H, 128, 32, generator=g) * 0.1).to(BF)
    QU = torch.bmm(q.float(), Uq.float()).to(BF)
    KU = torch.bmm(k.float(), Uq.float()).to(BF)
    ck0 = KU[:, torch.randperm(N, generator=g)[:2048].sort().values].contiguous()
    cq0 = QU[:, torch.randperm(N, generator=g)[:CQ].sort().values].contiguous()
    km = _kmm(lib, QU, KU, v, cq0, ck0, CQ)
    for ns in (491, 1638, 5):
        _select(lib, QU, km["cks16"], km["kcounts"], km["qperm"], km["qcounts"], ns)
        assert _select.requeued < 0.02 * H * N, (ns, _select.requeued)


@pytest.mark.parametrize("ns,pin_tail", [(204, 0), (1, 0), (4096, 0), (61, 33)])
def test_select_union_bit_exact(lib, small_case, ns, pin_tail):
    c = small_case
    QU = O.project(c["q"], c["state"]["Uq"], BF)
    KU = O.project(c["k"], c["state"]["Uk"], BF)
    km = O.kmeans_maintain(QU, KU, c["v"], c["state"]["cq"], c["state"]["ck"], pin_tail, BF)
    cks = (km["ck2"] * (1.0 / math.sqrt(128.0))).to(BF)
    want_u, want_rc = O.select_union(QU, cks, km["kcounts"], km["qlab"], c["CQ"], ns, pin_tail)
    got_u, got_rc = _select(lib, QU, cks, km["kcounts"], km["qperm"], km["qcounts"], ns, pin_tail)
    assert torch.equal(got_rc, want_rc)
    assert torch.equal(got_u, want_u)


def test_select_union_ties_and_empty_clusters(lib):
    """Small-integer scores tie massively; a third of the key clusters are empty,
    and one query cluster has no rows."""
    H, N, CQ, C = 1, 4096, 16, 2048
    g = torch.Generator().manual_seed(11)
    QU = torch.randint(-2, 3, (H, N, 32), generator=g).to(BF)
    cks = (torch.randint(-2, 3, (H, C, 32), generator=g).float() * 0.125).to(BF)
    klab = torch.randint(0, C, (H, N), generator=g).to(torch.int32)
    klab = torch.where(klab % 3 == 0, klab + 1, klab).clamp_max(C - 1)
    kcounts, _ = O.stable_group(klab, C)
    qlab = torch.randint(0, CQ - 1, (H, N), generator=g).to(torch.int32)      # cluster CQ-1 stays empty
    qcounts, qperm = O.stable_group(qlab, CQ)
    for ns in (40, 300):
        want_u, want_rc = O.select_union(QU, cks, kcounts, qlab, CQ, ns)
        got_u, got_rc = _select(lib, QU, cks, kcounts, qperm, qcounts, ns)
        assert torch.equal(got_rc, want_rc)
        assert torch.equal(got_u, want_u)
    assert int(got_u[0, CQ - 1].abs().sum()) == 0


def _tile_attn(lib, q, k, v, QU, km, cks, unip, tailw=1.0):
    H, N, _ = q.shape
    CQ = km["qcounts"].shape[1]
    kp = torch.gather(k, 1, km["kperm"].long()[..., None].expand(H, N, 128)).contiguous()
    plan = torch.zeros(lib.t2t_tile_attn_plan_ints(H, N, CQ), dtype=torch.int32, device=DEV)
    ws = torch.empty(lib.t2t_tile_attn_ws_bytes(H, N), dtype=torch.uint8, device=DEV)
    out = torch.zeros(H, N, 128, dtype=BF, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    tw = torch.tensor(float(tailw), dtype=torch.float32, device=DEV)
    host = [q, kp, km["V_sorted"], km["qcounts"], km["kcounts"], unip, QU, cks, km["sumv"], km["lam"], km["qlab"],
            km["qperm"]]
    dev = [t.to(DEV).contiguous() for t in host]
    _ok(lib.t2t_tile_attn(*[t.data_ptr() for t in dev], tw.data_ptr(), out.data_ptr(), plan.data_ptr(), 1, H, N,
                          CQ, ws.data_ptr(), ws.numel(), status.data_ptr(), _st()))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    info = torch.zeros(4, dtype=torch.int32, device=DEV)
    _ok(lib.t2t_tile_attn_plan_info(plan.data_ptr(), H, N, CQ, info.data_ptr(), _st()))
    i = info.cpu().tolist()
    lse = ws[((H * N * 256 + 255) // 256) * 256:].view(torch.float32)[: H * N].view(H, N).cpu()
    attn_o = ws[: H * N * 256].view(BF).view(H, N, 128).cpu()
    return out.cpu(), dict(tasks=i[0], pairs=(i[1] & 0xFFFFFFFF) | ((i[2] & 0xFFFFFFFF) << 32), lse=lse,
                           attn_o=attn_o)


def _structure(c, ns, pin_tail=0):
    QU = O.project(c["q"], c["state"]["Uq"], BF)
    KU = O.project(c["k"], c["state"]["Uk"], BF)
    km = O.kmeans_maintain(QU, KU, c["v"], c["state"]["cq"], c["state"]["ck"], pin_tail, BF)
    cks = (km["ck2"] * (1.0 / math.sqrt(128.0))).to(BF)
    unip, _ = O.select_union(QU, cks, km["kcounts"], km["qlab"], c["CQ"], ns, pin_tail)
    return QU, km, cks, unip


@pytest.mark.parametrize("kind", ["two humps", "heavy tails"])
def test_select_of_unlike_distributions_stays_on_the_tensor_core_path(lib, kind):
    """Half of the tokens around one centre (two humps of scores, the threshold in the upper one) and rows with Student
    tails: the first histogram range still brackets the threshold of nearly every row (measured 0.3 % and none queued for
    the exact kernel; half of the rows with a range of 1.6 deviations instead of 2.5)."""
    from token2tile_b200.deploy_step import MaskedStepDeploy
    H, N, CQ = 2, 16384, 128
    g = torch.Generator().manual_seed(9)
    rn = lambda *shape: torch.randn(*shape, generator=g)
    if kind == "two humps":
        pick = torch.where(torch.rand(N, generator=g) < 0.5, 0, torch.randint(0, 256, (N,), generator=g))
        base = rn(H, 256, 128)[:, pick]
        q, k = base + 0.3 * rn(H, N, 128), base + 0.3 * rn(H, N, 128)
    else:
        q, k = (rn(H, N, 128) / torch.sqrt((rn(H, N, 3) ** 2).mean(2, keepdim=True) + 0.05) for _ in range(2))
    q, k, v = (t.to(BF).to(DEV) for t in (q, k, rn(H, N, 128)))
    op = MaskedStepDeploy(H, N, CQ, s_frac=0.015)
    op.step(q, k, v, op.init_state(q, k, warm_iters=2))
    S = op.last_structure
    _select(lib, op.QU, S["cks"], S["counts"], S["qperm"], S["tile_sizes"], op.ns)
    assert _select.requeued <= 0.02 * H * N


@pytest.mark.parametrize("ns", [204, 20])
def test_tile_attn_matches_oracle(lib, small_case, ns):
    c = small_case
    scale = 1.0 / math.sqrt(128.0)
    QU, km, cks, unip = _structure(c, ns)
    o, lse = O.exact_attention(c["q"], c["k"], c["v"], km["qlab"], km["klab"], unip, scale)
    want = O.residual_merge(o, lse, QU, cks, km["sumv"], km["lam"], km["kcounts"], unip, km["qlab"], 1.0)
    got, info = _tile_attn(lib, c["q"], c["k"], c["v"], QU, km, cks, unip)
    # exact part, in sorted row order on the device
    perm = km["qperm"].long()
    o_sorted = torch.gather(o, 1, perm[..., None].expand_as(o))
    lse_sorted = torch.gather(lse, 1, perm)
    fin = torch.isfinite(lse_sorted)
    assert torch.equal(fin, torch.isfinite(info["lse"]))
    assert (info["lse"][fin] - lse_sorted[fin]).abs().max() < 2e-2
    assert (info["attn_o"].float() - o_sorted).abs().max() < 2e-2
    err = (got.float() - want).abs()
    assert err.max() < 2e-2, err.max()
    assert err.mean() < 2e-3, err.mean()
    kv = O.kv_lengths(unip, km["qcounts"], km["kcounts"])
    assert info["pairs"] == int((kv.long() * km["qcounts"].long()).sum())


def test_tile_attn_full_union_equals_dense(lib, small_case):
    """With every key cluster selected the operator is dense attention."""
    c = small_case
    QU, km, cks, unip = _structure(c, 204)
    full = torch.full_like(unip, -1)
    got, info = _tile_attn(lib, c["q"], c["k"], c["v"], QU, km, cks, full)
    want = O.dense_attention(c["q"], c["k"], c["v"], 1.0 / math.sqrt(128.0))
    err = (got.float() - want).abs()
    assert err.max() < 2e-2 and err.mean() < 2e-3
    assert info["pairs"] == c["H"] * c["N"] * c["N"]


def test_tile_attn_empty_union_is_pure_residual(lib, small_case):
    c = small_case
    QU, km, cks, unip = _structure(c, 204)
    none = torch.zeros_like(unip)
    got, info = _tile_attn(lib, c["q"], c["k"], c["v"], QU, km, cks, none)
    o = torch.zeros(c["H"], c["N"], 128)
    lse = torch.full((c["H"], c["N"]), -math.inf)
    want = O.residual_merge(o, lse, QU, cks, km["sumv"], km["lam"], km["kcounts"], none, km["qlab"], 1.0)
    err = (got.float() - want).abs()
    assert err.max() < 2e-2 and err.mean() < 2e-3
    assert info["pairs"] == 0


@pytest.mark.parametrize("H, N", [(1, 1), (2, 127), (3, 129), (1, 2048), (8, 9473), (2, 37889)])
@pytest.mark.parametrize("Cn", [1, 15, 17, 129, 512, 2048, 2050])
def test_assign_edges_of_tiles_groups_and_chunks(lib, H, N, Cn):
    """Few and many tiles, ragged rows, centroid counts around a group of 16 and a chunk of 128; a third of the centroids are copies of others - in the same group, in one other group, in many -
    and a few rows and centroids are not finite.  Labels equal the all-exact kernel's (checked by the helper)."""
    g = torch.Generator().manual_seed(N + Cn)
    cen = torch.randn(H, Cn, 32, generator=g)
    for c in range(0, Cn - 1, 3):
        cen[:, c + 1] = cen[:, c]                    # same group, mostly
    for c in range(2, Cn, 48):
        cen[:, c] = cen[:, (c + 16) % Cn]            # two groups
    cen[:, ::97] = cen[:, :1].clone()                # many groups
    if Cn > 100:
        cen[0, 77, 5] = float("inf")
    x = cen[:, torch.randint(0, Cn, (N,), generator=g)] + 0.2 * torch.randn(H, N, 32, generator=g)
    x[:, :: max(1, N // 7)] = cen[:, :1].clone()     # exact hits
    if N > 50:
        x[0, 33] = float("nan")
        x[0, 34, 2] = float("inf")
    _assign(lib, x.to(BF).to(DEV), cen.to(BF).to(DEV))
    finite = torch.nan_to_num(cen, posinf=1.0)       # and with finite centroids, where the bound does its work
    _assign(lib, x.to(BF).to(DEV), finite.to(BF).to(DEV))


@pytest.mark.parametrize("H, N", [(1, 130), (2, 4096), (1, 37889)])
@pytest.mark.parametrize("Cn", [48, 2048, 2050])
@pytest.mark.parametrize("kind", ["constant tail", "noisy tail", "all equal", "two families", "not finite"])
def test_assign_many_rows_near_many_equal_centroids(lib, H, N, Cn, kind):
    """Tiles full of rows with more than two groups in reach: a tail of equal rows (and of rows beside them) under centroids
    drawn from all rows, nothing but equal rows, two sets of equal centroids, and NaN and infinite rows and centroids.
    Labels equal the all-exact kernel's (checked by the helper)."""
    g = torch.Generator().manual_seed(N + Cn)
    x = torch.randn(H, N, 32, generator=g)
    tail = N if kind == "all equal" else max(100, N // 10)
    x[:, N - tail:] = x[:, -1:].clone()
    if kind == "two families":
        x[:, N - tail::2] = -x[:, -1:].clone()
    cen = x[:, torch.sort(torch.randint(0, N, (Cn,), generator=g)).values].clone()
    if kind == "two families":
        cen[:, ::3], cen[:, 1::3] = x[:, -1:].clone(), -x[:, -1:].clone()
    if kind == "noisy tail":
        x[:, N - tail:] += 1e-2 * torch.randn(H, tail, 32, generator=g)
    if kind == "not finite":
        x[:, N - 60:, 3] = float("nan")
        x[:, N - 90:N - 60, 4] = float("inf")
        cen[0, 5, 0] = float("inf")
        cen[0, 17, 1] = float("nan")
    _assign(lib, x.to(BF).to(DEV), cen.to(BF).to(DEV), pin_begin=N - 3, pin_label=1)


def test_assign_time_with_a_tail_of_equal_rows(lib):
    """Padding must not decide how long a call takes: with a tenth of the rows equal (and as many of the centroids), within
    eight times the call without (about three; settling such rows one by one takes twenty times as long)."""
    from token2tile_b200.deploy_step import fast_assign
    g = torch.Generator(device=DEV).manual_seed(4)
    N = 75600
    x = torch.randn(1, N, 32, device=DEV, generator=g)
    rows = torch.randperm(N, device=DEV, generator=g)[:2048].sort().values

    def time(x):
        x = x.to(BF)
        cen, out, ms = x[:, rows].contiguous(), torch.empty(1, N, dtype=torch.int32, device=DEV), []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(5):
                fast_assign(x, cen, out)
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
        return min(ms)

    plain = time(x)
    x[:, N - N // 10:] = x[:, -1:].clone()
    assert time(x) < 8.0 * plain


def _plain_structure(sizes, v):
    """One head, clusters of consecutive rows, every query cluster executes every key: (km, full union, zero QU)."""
    N, CQ = v.shape[1], len(sizes)
    ids = torch.arange(N, dtype=torch.int32)[None]
    km = dict(qcounts=torch.tensor([sizes], dtype=torch.int32), kcounts=torch.full((1, 2048), 2, dtype=torch.int32),
              qperm=ids, kperm=ids, qlab=torch.repeat_interleave(torch.arange(CQ), torch.tensor(sizes)).int()[None],
              V_sorted=v, sumv=torch.zeros(1, 2048, 128, dtype=BF), lam=torch.ones(1))
    return km, torch.full((1, CQ, 64), -1, dtype=torch.int32), torch.zeros(1, N, 32, dtype=BF)


@pytest.mark.parametrize("sizes", [(256, 129, 128, 127, 1, 3455 - 256 * 11), (4096,)])
def test_tile_attn_reference_maximum_far_below_later_scores(lib, sizes):
    """The reference of a row follows its maximum: scores that rise inside the first half of a tile (20, 40, 30 bits, the
    last one right behind a rise in the second half of the tile before), inside the second (70 and 140 bits: past the
    largest float), that fall by 200 bits and rise by 350, and that climb by 8 bits a tile, the step below which the
    reference stays; by the sign and size of q[0], rows of one warp see all of it, half, none, or all of it upside down.
    Against a float64 softmax of the same bfloat16 values; the weights are rounded to bfloat16 (2^-9 of values around 1,
    averaged) and so is the output."""
    N = 4096
    sizes = list(sizes) + [256] * 11 if len(sizes) > 1 else list(sizes)
    assert sum(sizes) == N
    g = torch.Generator().manual_seed(N + len(sizes))
    level = torch.zeros(N)
    for tile, pos, jump in ((2, 10, 20.0), (4, 3, 40.0), (6, 70, 70.0), (7, 20, 30.0), (9, 100, 140.0), (12, 0, -200.0),
                            (14, 20, 350.0)):
        level[tile * 128 + pos:] += jump
    level[16 * 128:] += 8.0 * (torch.arange(16 * 128) // 128)
    level += 2.0 * torch.randn(N, generator=g)
    k = 0.1 * torch.randn(1, N, 128, generator=g)
    k[0, :, 0] = level * math.sqrt(128.0) / math.log2(math.e) / 16.0
    q = 0.1 * torch.randn(1, N, 128, generator=g)
    q[0, :, 0] = 16.0 * torch.tensor([1.0, 0.5, 0.0, -1.0])[torch.randint(0, 4, (N,), generator=g)]
    v = torch.randn(1, N, 128, generator=g)
    q, k, v = q.to(BF), k.to(BF), v.to(BF)
    km, full, zeros = _plain_structure(sizes, v)
    _, info = _tile_attn(lib, q, k, v, zeros, km, zeros[:, :2048].contiguous(), full)
    s = q[0].double() @ k[0].double().T / math.sqrt(128.0)
    want = torch.softmax(s, 1) @ v[0].double()
    assert (info["attn_o"][0].double() - want).abs().max() < 2e-2
    assert (info["lse"][0].double() - torch.logsumexp(s, 1)).abs().max() < 1e-2


@pytest.mark.parametrize("sizes", [(4096,), (128,) * 32])
@pytest.mark.parametrize("tile, pos", [(0, 3), (5, 20), (5, 100), (31, 127)])
def test_tile_attn_weight_of_a_dominant_key_is_one(lib, sizes, tile, pos):
    """One key 45 to 56 bits above all others, in the first or second half of an early or late tile, and values of 1e30:
    its weight is exactly one in bfloat16, so the output is its value bit for bit (the other 4,095 weigh 2^-33 together)
    and nothing between them leaves the range of fp32."""
    N = 4096
    g = torch.Generator().manual_seed(tile)
    q, k = torch.zeros(1, N, 128), torch.zeros(1, N, 128)
    q[0, :, 0] = 16.0 + (torch.arange(N) % 32) / 8.0
    k[0, tile * 128 + pos, 0] = 22.0
    v = (1.0 + torch.rand(1, N, 128, generator=g)) * torch.where(torch.rand(1, N, 128, generator=g) < 0.5, -1e30, 1e30)
    q, k, v = q.to(BF), k.to(BF), v.to(BF)
    km, full, zeros = _plain_structure(list(sizes), v)
    _, info = _tile_attn(lib, q, k, v, zeros, km, zeros[:, :2048].contiguous(), full)
    assert torch.equal(info["attn_o"][0], v[0, tile * 128 + pos].expand(N, 128))
    s = q[0].double() @ k[0].double().T / math.sqrt(128.0)
    assert (info["lse"][0].double() - torch.logsumexp(s, 1)).abs().max() < 1e-4


def _unions_of_many_forms(largest):
    """(key cluster sizes, query cluster sizes, selected clusters, the same as bitmaps, generator) of twelve heads."""
    H, N = 12, 6000
    g = torch.Generator().manual_seed(largest)
    kc = torch.zeros(H, 2048, dtype=torch.int32)
    for h in range(H):
        kc[h, :600] = 1
        kc[h, 600:1200] = torch.randint(0, 4, (600,), generator=g).int()
        kc[h, 1200] = 128
        kc[h, 1202:1220] = torch.randint(30, 140, (18,), generator=g).int()
        kc[h, 2047] = N - int(kc[h].sum())
    assert int(kc.min()) == 0 and int(kc[:, 2047].min()) > 256
    edge = [1, 31, 32, 33, 64, 127, 128] + ([129, 160, 255, 256, 257, 300] if largest > 128 else [])
    sizes = list(edge)
    while N - sum(sizes) > largest:
        sizes.append(int(torch.randint(1, largest + 1, (1,), generator=g)))
    sizes.append(N - sum(sizes))
    CQ = len(sizes)
    sel = torch.zeros(H, CQ, 2048, dtype=torch.bool)
    for h in range(H):
        for c in range(CQ):
            kind = (c + h) % 10
            if kind == 1: sel[h, c, 5] = True
            elif kind in (2, 3, 4): sel[h, c, 7:7 + 127 + (kind - 2)] = True
            elif kind == 5: sel[h, c, 0:600:2] = True
            elif kind == 6: sel[h, c, 600:1200:2] = True
            elif kind == 7: sel[h, c, [3, 1200, 1203, 1204, 1205, 1210, 2047]] = True
            elif kind == 8: sel[h, c] = True
            elif kind == 9: sel[h, c] = torch.rand(2048, generator=g) < 0.2
            if kind == 4 and c % 2: sel[h, c, 1200] = True
    bits = (sel.view(H, CQ, 64, 32).long() << torch.arange(32)).sum(-1)
    union = torch.where(bits >= 2 ** 31, bits - 2 ** 32, bits).int()
    return kc, sizes, sel, union, g


@pytest.mark.parametrize("largest", [128, 300])
def test_tile_attn_unions_of_many_forms(lib, largest):
    """Tasks of 1 to `largest` rows, several to a CTA, with unions of no key, of one, of 127 / 128 / 129 / 256, of clusters
    of one key each with gaps (more than 32 runs in a tile), of long stretches at odd offsets, of everything; empty
    clusters inside.  Against a float64 softmax over the union: the weights and the output are rounded to bfloat16."""
    kc, sizes, sel, union, g = _unions_of_many_forms(largest)
    H, N = len(kc), sum(sizes)
    q, k, v = (torch.randn(H, N, 128, generator=g).to(BF) for _ in range(3))
    km, _, zeros = _plain_structure(sizes, v[:1])
    km = {key: t.expand(H, *t.shape[1:]).contiguous() for key, t in km.items() if key != "lam"}
    km.update(lam=torch.ones(H), kcounts=kc, V_sorted=v)
    _, info = _tile_attn(lib, q, k, v, torch.zeros(H, N, 32, dtype=BF), km, torch.zeros(H, 2048, 32, dtype=BF), union)
    lab = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes))
    for h in range(H):
        inside = torch.repeat_interleave(sel[h], kc[h].long(), dim=1)[lab].to(DEV)
        s = q[h].to(DEV).double() @ k[h].to(DEV).double().T / math.sqrt(128.0)
        s = torch.where(inside, s, -math.inf)
        some = inside.any(1)
        want = torch.where(some[:, None], torch.softmax(s, 1), 0.0) @ v[h].to(DEV).double()
        lse = torch.logsumexp(s, 1).cpu()
        assert (info["attn_o"][h].double() - want.cpu()).abs().max() < 2e-2
        fin = some.cpu()
        assert torch.equal(torch.isfinite(info["lse"][h]), fin)
        assert (info["lse"][h].double() - lse)[fin].abs().max() < 1e-2


@pytest.mark.parametrize("largest", [128, 300])
def test_tile_attn_meets_every_row_of_a_union_once(lib, largest):
    """The same unions, with keys and values that show a row that is missing, read twice or taken from its neighbour, however
    long the union is: in an average of thousands of normal values one row for another moves an output by 6e-3 at most, less
    than the bound above.

    Values: q = 0, so every weight is one and the output is what a union holds of each of 128 codes (a random one per key,
    one-hot), divided by its length: whole numbers below 2^24, so the same bits as the count rounded once each by the
    division, the product and bfloat16.  Keys: a code's score is 8 / log2(e) or 0, by random bits of the query, so that
    one key for another of other score changes its logsumexp by a 6000th or more (fp32 sums 6,000 weights to within 1e-5 and
    rounds the result to 1e-6)."""
    kc, sizes, sel, union, g = _unions_of_many_forms(largest)
    H, N = len(kc), sum(sizes)
    code = torch.randint(0, 128, (H, N), generator=g)
    onehot = torch.nn.functional.one_hot(code, 128)
    km, _, _ = _plain_structure(sizes, torch.zeros(1, N, 128, dtype=BF))
    km = {key: t.expand(H, *t.shape[1:]).contiguous() for key, t in km.items() if key != "lam"}
    km.update(lam=torch.ones(H), kcounts=kc, V_sorted=onehot.to(BF))
    rest = torch.zeros(H, N, 32, dtype=BF), km, torch.zeros(H, 2048, 32, dtype=BF), union
    # per query cluster: which keys its union holds, and how many of each code
    keys = torch.stack([torch.repeat_interleave(sel[h], kc[h].long(), dim=1) for h in range(H)])
    counts = keys.float() @ onehot.float()
    length = keys.sum(-1)
    lab = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes))
    average = lambda counts, length: (counts * (1.0 / length.clamp(min=1).float())[..., None]).to(BF)
    _, info = _tile_attn(lib, torch.zeros(H, N, 128, dtype=BF), torch.randn(H, N, 128, generator=g).to(BF),
                         km["V_sorted"], *rest)
    assert torch.equal(info["attn_o"], average(counts, length)[:, lab])

    q = 16.0 * torch.randint(0, 2, (H, N, 128), generator=g).to(BF)
    k = onehot.to(BF) * (8.0 * math.log(2.0) * math.sqrt(128.0) / 16.0)
    _, info = _tile_attn(lib, q, k, km["V_sorted"], *rest)
    weight = torch.exp(q.double() * float(k.max()) / math.sqrt(128.0))      # of a key by its code
    lse = lambda counts: (counts.double()[:, lab] * weight).sum(-1).log()
    some = length[:, lab] > 0
    assert torch.equal(torch.isfinite(info["lse"]), some)
    assert (info["lse"].double() - lse(counts))[some].abs().max() < 2e-5

    # both would see one key of the longest union replaced by its neighbour
    long = (length == N) & (torch.tensor(sizes) > 8)
    a = 2 * N // 3
    b = a + 1 + int((code[:, a + 1:] != code[:, a:a + 1]).long().argmax(1).max())
    wrong = counts - onehot[:, None, a] + onehot[:, None, b]
    moved = (code[:, a] != code[:, b])[:, None] & long
    assert bool(moved.any()) and bool((average(wrong, length) != average(counts, length)).any(-1)[moved].all())
    moved = moved[:, lab]
    change = (lse(wrong) - lse(counts)).abs()
    assert float((change > 4e-5)[moved].double().mean()) > 0.3


@pytest.mark.parametrize("N", [31, 257, 8192, 8193, 16384, 16385])
@pytest.mark.parametrize("Cn", [3, 1024, 2048])
def test_centroid_update_on_both_sides_of_the_chunk_rule(lib, N, Cn):
    """256 rows per warp up to 16,384 rows (8,192 above 1024 clusters), 1024 beyond; ragged ends, labels outside [0, Cn) left out, empty clusters
    keeping their old centroid.  The sums are exact integers: bit for bit."""
    H = 2
    g = torch.Generator().manual_seed(N + Cn)
    x = torch.randn(H, N, 32, generator=g).to(BF)
    lab = torch.randint(-1, Cn + 1, (H, N), generator=g).int()
    old = torch.randn(H, Cn, 32, generator=g).to(BF)
    fixed = torch.round(x.double() * 32768.0).long()
    inside = (lab >= 0) & (lab < Cn)
    sums, counts = torch.zeros(H, Cn + 1, 32, dtype=torch.long), torch.zeros(H, Cn + 1, dtype=torch.long)
    idx = torch.where(inside, lab, Cn).long()
    for h in range(H):
        sums[h].index_add_(0, idx[h], fixed[h])
        counts[h] = torch.bincount(idx[h], minlength=Cn + 1)
    counts = counts[:, :Cn]
    want = (sums[:, :Cn].float() / (32768.0 * counts.float())[..., None]).to(BF)
    want = torch.where(counts[..., None] > 0, want, old)
    newc = torch.empty(H, Cn, 32, dtype=BF, device=DEV)
    got_counts = torch.empty(H, Cn, dtype=torch.int32, device=DEV)
    ws = torch.empty(lib.t2t_centroid_update_ws_bytes(H, N, Cn), dtype=torch.uint8, device=DEV)
    xd, ld, od = x.to(DEV), lab.to(DEV), old.to(DEV)
    _ok(lib.t2t_centroid_update(xd.data_ptr(), ld.data_ptr(), od.data_ptr(), newc.data_ptr(), got_counts.data_ptr(), H, N,
                                Cn, ws.data_ptr(), ws.numel(), _st()))
    torch.cuda.synchronize()
    assert torch.equal(got_counts.cpu().long(), counts)
    assert torch.equal(newc.cpu(), want)


@pytest.mark.parametrize("H, N, CQ", [(1, 2049, 1), (2, 4096, 300), (5, 31000, 97), (40, 15361, 40)])
@pytest.mark.parametrize("share", [0.0005, 0.015, 0.3])
def test_select_tiles_per_cta_and_ragged_tiles(lib, H, N, CQ, share):
    """One, two and eight tiles per CTA (the last one ragged, and the last CTA short), tiles inside one query cluster
    and tiles spanning many, tiny and large budgets: the same unions and token counts as the all-exact kernel."""
    g = torch.Generator().manual_seed(N)
    centres = torch.randn(H, 60, 32, generator=g)
    pick = lambda n: centres[:, torch.randint(0, 60, (n,), generator=g)]
    QU = (pick(N) + 0.3 * torch.randn(H, N, 32, generator=g)).to(BF)
    cks = (0.1 * (pick(2048) + 0.3 * torch.randn(H, 2048, 32, generator=g))).to(BF)
    counts = torch.bincount(torch.randint(0, 2048, (N,), generator=g), minlength=2048).int()[None].expand(H, -1).contiguous()
    qlab = torch.randint(0, CQ, (H, N), generator=g)
    qcounts = torch.stack([torch.bincount(q, minlength=CQ) for q in qlab]).int()
    qperm = torch.sort(qlab, dim=1, stable=True).indices.int()
    _select(lib, QU, cks, counts, qperm, qcounts, max(1, int(share * N)))
