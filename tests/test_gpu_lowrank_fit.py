"""The projection-fit kernels (t2t_lowrank_fit: tensor-core second moments, fp64
factors and singular triplets) against the reference's own `online_u` run on the CPU
(tests/golden/online_u.pt) and against the oracle.

The factors are defined up to a common sign per component (and a rotation
inside equal singular values), so the products Uq Uk^T are compared; one test
pins the signs that the order of the rotations gives them."""
import importlib.util
from pathlib import Path

import pytest
import torch

from oracle import t2t_oracle as O

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
DEV = "cuda"
GOLDEN = Path(__file__).resolve().parent / "golden"


def _product(Uq, Uk):
    return Uq.double().cpu() @ Uk.double().cpu().transpose(1, 2)


def _golden_inputs():
    spec = importlib.util.spec_from_file_location("mk", GOLDEN / "make_online_u_golden.py")
    mk = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mk)
    return mk


def test_fit_matches_the_reference_golden_vectors():
    """The golden inputs are fp32; the kernels take them rounded to bfloat16 (a relative
    perturbation of 2^-9 per element), which bounds the agreement."""
    from token2tile_b200.deploy_step import online_u
    mk = _golden_inputs()
    for item in torch.load(GOLDEN / "online_u.pt"):
        q, k = mk.make_inputs(item["case"])
        Uq, Uk = online_u(q.to(DEV), k.to(DEV), item["case"]["r"])
        want = _product(item["Uq"], item["Uk"])
        got = _product(Uq, Uk)
        assert (got - want).abs().max() <= 2e-2 * want.abs().max(), item["case"]
        # and tightly against the oracle given the very same bfloat16 values
        qb, kb = q.to(BF).float(), k.to(BF).float()
        oq, ok = O.online_u(qb, kb, item["case"]["r"])
        want_b = _product(oq, ok)
        assert (got - want_b).abs().max() <= 1e-4 * want_b.abs().max(), item["case"]


@pytest.mark.parametrize("N", [4096, 20001])
def test_fit_matches_the_oracle_on_bfloat16_inputs(N):
    """N = 20,001: three slabs of the Gram kernel and a ragged last tile."""
    from token2tile_b200.deploy_step import online_u
    from token2tile_b200.t2t_attn import fast_online_u
    g = torch.Generator().manual_seed(21)
    H = 3
    k = (torch.randn(H, N, 128, generator=g) * torch.linspace(2.0, 0.05, 128)).to(BF)
    q = (0.6 * k.float() + 0.4 * torch.randn(H, N, 128, generator=g) * torch.linspace(0.05, 2.0, 128)).to(BF)
    Uq, Uk = online_u(q.to(DEV), k.to(DEV), 32)
    assert Uq.dtype == torch.float32 and Uq.shape == (H, 128, 32)
    oq, ok = O.online_u(q.float(), k.float(), 32)
    want, got = _product(oq, ok), _product(Uq, Uk)
    assert (got - want).abs().max() <= 1e-4 * want.abs().max()
    # the logit approximation the projections exist for
    err = ((q.double() @ got) @ k.double().transpose(1, 2) - (q.double() @ want) @ k.double().transpose(1, 2))[:, :256, :256]
    assert err.abs().max() <= 1e-3 * (q.double() @ k.double().transpose(1, 2))[:, :256, :256].abs().max()
    fq, fk = fast_online_u(q.to(DEV), k.to(DEV), 32)       # same kernels, no finiteness read-back
    torch.cuda.synchronize()
    assert torch.equal(fq, Uq) and torch.equal(fk, Uk)


def test_fit_of_rank_deficient_inputs():
    """Queries confined to a 20-dimensional subspace: 108 clamped eigenvalues on the query side and
    fewer than 32 non-zero singular values."""
    from token2tile_b200.deploy_step import online_u
    g = torch.Generator().manual_seed(22)
    basis = torch.linalg.qr(torch.randn(128, 20, generator=g)).Q
    q = ((torch.randn(2, 3000, 20, generator=g) @ basis.T)).to(BF)
    k = torch.randn(2, 3000, 128, generator=g).to(BF)
    Uq, Uk = online_u(q.to(DEV), k.to(DEV), 32)
    assert bool(torch.isfinite(Uq).all()) and bool(torch.isfinite(Uk).all())
    logits = q.double() @ k.double().transpose(1, 2)
    approx = (q.double() @ _product(Uq, Uk)) @ k.double().transpose(1, 2)
    oq, ok = O.online_u(q.float(), k.float(), 32)
    approx_o = (q.double() @ _product(oq, ok)) @ k.double().transpose(1, 2)
    # rank 20 < 32: the fit reproduces the logits, as the oracle's does
    assert (approx - logits).abs().max() <= 1e-2 * logits.abs().max()
    assert (approx - approx_o).abs().max() <= 1e-2 * logits.abs().max()


def test_fit_rejects_non_finite_inputs():
    from token2tile_b200.deploy_step import online_u
    from token2tile_b200.t2t_attn import fast_online_u
    g = torch.Generator().manual_seed(23)
    q = torch.randn(2, 1024, 128, generator=g).to(BF).to(DEV)
    k = q.clone()
    k[1, 7, 3] = float("inf")
    with pytest.raises(RuntimeError, match="non-finite k input in heads \\[1\\]"):
        online_u(q, k, 32)
    fq, fk = fast_online_u(q, k, 32)          # no exception: the bad head's projections stay zero
    torch.cuda.synchronize()
    assert bool((fq[1] == 0).all()) and bool((fk[1] == 0).all()) and bool(fq[0].abs().sum() > 0)
    with pytest.raises(ValueError):
        online_u(q, k, 16)


@pytest.mark.parametrize("N", [2048, 2177, 8192 + 1])
@pytest.mark.parametrize("spread_q, spread_k", [(1.0, 1.0), (3e-3, 1.0), (1e-6, 3e-3), (1.0, 1e-6), (1.0, 0.3), (0.3, 0.03)])
def test_fit_on_both_factor_routes(N, spread_q, spread_k):
    """Cholesky factor, root by products and clamped root by eigenvectors, with condition numbers of the key side
    from 2 to 1e12 (the products give up in between) and both sides on either side of the clamp: smallest moments of
    0.3 and 4e-6 (Cholesky: the trace of the inverse is 3e6) and of 5e-13 (below the clamp).  Several and ragged slabs.
    The oracle works in float64 on the same bfloat16 values; the kernels' second moments are fp32 sums per slab
    (2^-24 per addition, 2^-17 for a slab of thousands of rows at worst), and the fit divides by the gap between
    the singular values 32 and 33 (a quarter and more here): 1e-3 of the largest logit, as above."""
    from token2tile_b200.deploy_step import online_u
    g = torch.Generator().manual_seed(N)
    H = 2
    ramp = torch.linspace(0.0, 1.0, 128)
    step = torch.where(torch.arange(128) < 32, 1.0, 0.7)      # a gap between the kept and the dropped values
    mix = torch.block_diag(torch.linalg.qr(torch.randn(64, 64, generator=g)).Q, torch.eye(64))      # bfloat16 keeps the small ones
    q = ((torch.randn(H, N, 128, generator=g) * step * spread_q ** ramp) @ mix.T).to(BF)
    k = ((torch.randn(H, N, 128, generator=g) * step * spread_k ** ramp) @ mix.T).to(BF)
    Uq, Uk = online_u(q.to(DEV), k.to(DEV), 32)
    oq, ok = O.online_u(q.double(), k.double(), 32)
    # the logits' approximation is what is determined: clamped directions carry no data
    want = (q.double() @ _product(oq, ok)) @ k.double().transpose(1, 2)
    got = (q.double() @ _product(Uq, Uk)) @ k.double().transpose(1, 2)
    assert (got - want).abs().max() <= 1e-3 * want.abs().max()


@pytest.mark.parametrize("p", [4, 8, 10])
def test_fit_separates_nearly_equal_singular_values(p):
    """Second moments that fp32 slabs hold exactly: 8,192 Hadamard rows (one slab, 8192 I) and, on the query side, 300
    rows of integers times 2^-p (the next slab).  All singular values agree to 7e-4, 3e-6 and 2e-7; the 32 largest span
    a subspace that is determined to the fp64 rounding over the gap behind them (2^-52 x 128 over 5e-6, 1e-8 and 1e-9),
    plus the rounding of the fp32 factors."""
    from token2tile_b200.deploy_step import online_u
    had = torch.ones(1, 1)
    while had.shape[0] < 8192:
        had = torch.cat([torch.cat([had, had], 1), torch.cat([had, -had], 1)])
    had = had[:, torch.arange(128) * 64 + 1]
    assert torch.equal(had.double().T @ had.double(), 8192 * torch.eye(128).double())
    R = torch.randint(-2, 3, (300, 128), generator=torch.Generator().manual_seed(p)).float()
    q = torch.cat([had, R * 2.0 ** -p])[None].to(BF)
    k = torch.cat([had, torch.zeros(300, 128)])[None].to(BF)
    Uq, Uk = online_u(q.to(DEV), k.to(DEV), 32)
    e, V = torch.linalg.eigh(R.double().T @ R.double())
    want = V[:, -32:] @ V[:, -32:].T                  # Mq, Mk and their roots share these eigenvectors
    gap = float(e[-32] - e[-33]) * 4.0 ** -p / 8192 / 2
    got = _product(Uq, Uk)[0]
    assert (got - want).abs().max() <= (2.0 ** -52 * 128 / gap + 2.0 ** -22) * want.abs().max()


def test_rotation_against_float64(lib):
    """Angles from 1e-12 to 45 degrees, both signs, lengths that agree and that differ by 2^30.  t0 is within a few fp32
    roundings (3.2e-7 at worst) and the Newton step leaves their square and, in its own correction, another 1e-7 of
    them: 1e-12 covers it with room.  (c, s) is a rotation to fp64 rounding."""
    n = 1 << 16
    g = torch.Generator().manual_seed(3)
    u = lambda lo, hi: lo + (hi - lo) * torch.rand(n, generator=g, dtype=torch.float64)
    alpha, beta = 2.0 ** u(30, 60), 2.0 ** u(30, 60)
    beta = torch.where(torch.arange(n) % 3 == 0, alpha * (1.0 + 2.0 ** u(-40, 0)), beta)
    gamma = torch.sqrt(alpha * beta) * 10.0 ** u(-13, 0) * torch.where(torch.arange(n) % 2 == 0, 1.0, -1.0)
    pairs = torch.stack([alpha, beta, gamma], 1).to(DEV)
    out = torch.empty_like(pairs)
    assert lib.t2t_rotation_selftest(pairs.data_ptr(), out.data_ptr(), n, torch.cuda.current_stream().cuda_stream) == 0
    t, c, s = out.cpu().unbind(1)
    zeta = (beta - alpha) / (2.0 * gamma)
    want = torch.where(zeta >= 0, 1.0, -1.0) / (zeta.abs() + torch.sqrt(1.0 + zeta * zeta))
    assert ((t - want) / want).abs().max() < 1e-12
    assert (c * c + s * s - 1.0).abs().max() < 1e-15
    assert (s - c * t).abs().max() < 1e-15


def _factors(lib, q, k):
    """(Uq, Uk, roots [2 H, 128, 128]): the fit by its C entry, with the factors that it left in the workspace."""
    H, N, _ = q.shape
    qd, kd = q.to(DEV), k.to(DEV)
    U = torch.empty(2, H, 128, 32, device=DEV)
    flags = torch.zeros(2 * H + 1, dtype=torch.int32, device=DEV)
    ws = torch.empty(lib.t2t_lowrank_fit_ws_bytes(H, N), dtype=torch.uint8, device=DEV)
    assert lib.t2t_lowrank_fit(qd.data_ptr(), kd.data_ptr(), U[0].data_ptr(), U[1].data_ptr(), H, N, ws.data_ptr(), ws.numel(),
                               flags.data_ptr(), flags.data_ptr() + 8 * H, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert not bool(flags.any())
    at = ws.numel() - 3 * H * 128 * 128 * 8            # the last two regions: roots of 2 H matrices, inverses of H
    return U[0].cpu(), U[1].cpu(), ws[at:at + 2 * H * 128 * 128 * 8].view(torch.float64).view(2 * H, 128, 128).cpu()


@pytest.mark.parametrize("spread_q, spread_k, route_q, route_k", [
    (1.0, 1.0, "cholesky", "products"), (3e-3, 0.3, "cholesky", "products"), (0.3, 0.1, "cholesky", "products"),
    (1e-6, 1e-6, "eigenvectors", "eigenvectors")])
def test_fit_takes_the_factor_route_of_its_spread(lib, spread_q, spread_k, route_q, route_k):
    """The factor shows its route: Cholesky leaves zeros above the diagonal, the products end by averaging the root with
    its transpose (symmetric bit for bit), and the sum over eigenvectors rounds the two triangles differently.  All of
    them satisfy F F^T = M to the clamp and to the fp32 sums of the second moments: 256 additions of 16 rows each, every
    one off by at most 2^-23 of the sum."""
    g = torch.Generator().manual_seed(31)
    H, N = 2, 4096
    ramp = torch.linspace(0.0, 1.0, 128)
    mix = torch.block_diag(torch.linalg.qr(torch.randn(64, 64, generator=g)).Q, torch.eye(64))
    make = lambda spread: ((torch.randn(H, N, 128, generator=g) * spread ** ramp) @ mix.T).to(BF)
    q, k = make(spread_q), make(spread_k)
    _, _, F = _factors(lib, q, k)

    def route(f):
        if not bool(torch.triu(f, 1).any()):
            return "cholesky"
        return "products" if torch.equal(f, f.T) else "eigenvectors"

    assert [route(F[i]) for i in range(H)] == [route_q] * H
    assert [route(F[H + i]) for i in range(H)] == [route_k] * H
    x = torch.cat([q, k]).double()
    M = x.transpose(1, 2) @ x / N
    assert (F @ F.transpose(1, 2) - M).abs().max() < 256 * 2.0 ** -23 * M.abs().max() + 1e-8


def test_fit_signs_are_those_of_symmetric_roots(lib):
    """The factors come with the signs (and the order) that one-sided Jacobi gives for symmetric roots on both sides:
    round-robin rounds over M_q^(1/2) M_k^(1/2), restated here in float64.  Small integers, so that the second moments
    are the same numbers."""
    g = torch.Generator().manual_seed(32)
    N = 4096
    wide = torch.linspace(6.0, 1.0, 128)
    k = torch.round(torch.randn(N, 128, generator=g) * wide[torch.randperm(128, generator=g)])
    q = torch.round(0.5 * k + torch.randn(N, 128, generator=g) * wide)
    assert q.abs().max() < 256 and k.abs().max() < 256            # exact in bfloat16
    Uq, Uk, _ = _factors(lib, q[None].to(BF), k[None].to(BF))

    def powers(x):
        e, V = torch.linalg.eigh(x.double().T @ x.double() / N)
        return (V * e.sqrt()) @ V.T, (V / e.sqrt()) @ V.T

    (Rq, Iq), (Rk, _) = powers(q), powers(k)
    W = Rq @ Rk
    i = torch.arange(1, 64)
    for sweep in range(14):
        for r in range(127):
            x = torch.cat([torch.tensor([127]), (r + i) % 127])
            y = torch.cat([torch.tensor([r]), (r + 127 - i) % 127])
            a, b, c = (W[:, x] ** 2).sum(0), (W[:, y] ** 2).sum(0), (W[:, x] * W[:, y]).sum(0)
            turn = c * c > 1e-27 * a * b
            zeta = (b - a) / (2.0 * torch.where(turn, c, torch.ones(())))
            t = torch.where(zeta >= 0, 1.0, -1.0) / (zeta.abs() + torch.sqrt(1.0 + zeta * zeta)) * turn
            cos = 1.0 / torch.sqrt(1.0 + t * t)
            W[:, x], W[:, y] = cos * W[:, x] - cos * t * W[:, y], cos * t * W[:, x] + cos * W[:, y]
    s, order = torch.sort((W * W).sum(0).sqrt(), descending=True, stable=True)
    w, s = W[:, order[:32]], s[:32]
    want_q, want_k = Iq @ w / s.sqrt(), Rq @ w / (s * s.sqrt())
    for got, want in ((Uq[0], want_q), (Uk[0], want_k)):
        assert (got.double() - want).abs().max() < 1e-5 * want.abs().max()
