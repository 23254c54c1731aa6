"""Team sizes: a problem is solved by one CTA or by a cluster of up to 16 (few
problems in a call), and the results are the same bits either way; products
split over CTAs by output tiles."""
import ctypes

import numpy as np
import pytest

from libnegf_b200 import generators as G
from libnegf_b200 import native

pytestmark = pytest.mark.gpu


def _dp(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _ip(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_int32))


@pytest.mark.parametrize("dev", [
    lambda: G.transport_c0(nbl=3, n=33, seed=1),
    lambda: G.transport_c0(nbl=3, n=65, seed=1),                  # first order with leaves
    lambda: G.transport_c1(nbl=3, n=129, seed=2),                 # one row and column past two tiles
    lambda: G.uneven([40, 90, 17, 70], seed=3),
], ids=["n33", "n65", "n129_S", "uneven"])
def test_engine_results_do_not_depend_on_the_team_size(gpu_ctx, dev):
    did = gpu_ctx.upload(dev())
    E = np.linspace(-1.5, 1.5, 300)                                # more points than CTAs: teams of one
    try:
        T, nc, st = gpu_ctx.transmission(did, E, eta=1e-3)
        Td, dos, _, _ = gpu_ctx.transmission_dos(did, E, eta=1e-3, dos_delta=1e-3)
        for m in (1, 30, 80):                                      # teams of up to 16, 8 and 2 .. 4
            a = gpu_ctx.transmission(did, E[:m], eta=1e-3)
            b = gpu_ctx.transmission_dos(did, E[:m], eta=1e-3, dos_delta=1e-3)
            assert np.array_equal(a[0], T[:m]) and np.array_equal(a[1], nc[:m]) and np.array_equal(a[2], st[:m])
            assert np.array_equal(b[0], Td[:m]) and np.array_equal(b[1], dos[:m])
    finally:
        gpu_ctx.release(did)


@pytest.mark.parametrize("n", [64, 65, 96, 127, 129, 256, 257, 513])
def test_inverse_bits_do_not_depend_on_the_team_size(n):
    torch = pytest.importorskip("torch")
    L = native.load()
    batch = 300 if n <= 256 else 60
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((batch, n, n), dtype=torch.complex128, device="cuda", generator=g)
    X, X1 = torch.zeros_like(A), torch.zeros_like(A[:1])
    info = torch.full((batch,), -1, dtype=torch.int32, device="cuda")
    work = torch.empty(L.negf_b200_zinv_work_bytes(batch, n), dtype=torch.uint8, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    w = ctypes.c_void_p(work.data_ptr())
    assert L.negf_b200_zinv_batched(batch, n, _dp(A), _dp(X), _ip(info), w, s) == 0
    assert int(info.abs().max()) == 0
    assert L.negf_b200_zinv_batched(1, n, _dp(A), _dp(X1), _ip(info), w, s) == 0
    torch.cuda.synchronize()
    assert torch.equal(X1[0], X[0])
    A[0, :, 3] = 0.0                                               # a zero row: an exact zero pivot, seen by every member
    assert L.negf_b200_zinv_batched(1, n, _dp(A), _dp(X1), _ip(info), w, s) == 0
    torch.cuda.synchronize()
    assert int(info[0]) > 0


@pytest.mark.parametrize("m,n,k,batch", [(1, 1, 1, 1), (64, 65, 17, 2), (63, 130, 64, 1), (300, 20, 33, 5),
                                         (129, 129, 129, 200)])
@pytest.mark.parametrize("dagger", [0, 1, 2])
def test_split_products(m, n, k, batch, dagger):
    """Against torch: each side's rounding of a K-term complex sum is within
    2 (K + 2) u |A||B| elementwise."""
    torch = pytest.importorskip("torch")
    L = native.load()
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    r = lambda *s: torch.randn(s, dtype=torch.complex128, device="cuda", generator=g)
    A = r(batch, m, k) if dagger == 1 else r(batch, k, m)         # column major: reversed index order
    B = r(batch, k, n) if dagger == 2 else r(batch, n, k)
    C = torch.zeros((batch, n, m), dtype=torch.complex128, device="cuda")
    one, zero = (ctypes.c_double * 2)(1, 0), (ctypes.c_double * 2)(0, 0)
    rc = L.negf_b200_zgemm_batched(batch, m, n, k, one, _dp(A), 2 * m * k, _dp(B), 2 * k * n, zero, _dp(C),
                                   2 * m * n, dagger, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    a = A.conj() if dagger == 1 else A.transpose(1, 2)
    b = B.conj() if dagger == 2 else B.transpose(1, 2)
    err = (C.transpose(1, 2) - a @ b).abs()
    bound = 4 * (k + 2) * 2.0 ** -53 * (a.abs() @ b.abs())
    torch.cuda.synchronize()
    assert bool((err <= bound).all())


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 128, 129, 255, 256, 257, 511, 512, 513])
def test_inverse_at_the_panel_edges(n):
    """Against LAPACK on well-conditioned matrices: the residual A X - I of
    Gauss-Jordan with partial pivoting is within c(n) u kappa(A), with c(n)
    at most 8 n (n terms per entry, a few roundings each); rows in reverse
    order make every pivot an exchange, equal rows up to sign make ties."""
    torch = pytest.importorskip("torch")
    L = native.load()
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((3, n, n), dtype=torch.complex128, device="cuda", generator=g) / max(1.0, n ** 0.5)
    A = A + 4.0 * torch.eye(n, dtype=A.dtype, device="cuda")
    A[1] = A[1].flip(1)                                            # column major: rows reversed
    if n > 2:
        A[2] = torch.eye(n, dtype=A.dtype, device="cuda").flip(1) * 2.0
        A[2, :, 0] = 1.0                                           # a row of ties with the entries below
        A[2, 0, :] = 1.0
        A[2] += 3.0 * torch.eye(n, dtype=A.dtype, device="cuda")
    X = torch.zeros_like(A)
    info = torch.full((3,), -1, dtype=torch.int32, device="cuda")
    work = torch.empty(L.negf_b200_zinv_work_bytes(3, n), dtype=torch.uint8, device="cuda")
    assert L.negf_b200_zinv_batched(3, n, _dp(A), _dp(X), _ip(info), ctypes.c_void_p(work.data_ptr()),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert int(info.abs().max()) == 0
    for q in range(3):
        a = A[q].cpu().numpy().T
        x = X[q].cpu().numpy().T
        k = np.linalg.cond(a)
        assert np.abs(a @ x - np.eye(n)).max() <= 8 * n * 2.0 ** -53 * max(k, 1.0)


@pytest.mark.parametrize("n", [20, 50, 100, 200, 400])
def test_inverse_of_non_finite_matrices(n):
    """NaN never wins a pivot search and reaches the result; an infinite
    diagonal entry is a pivot whose reciprocal is 0: its row and column of
    the inverse vanish and the rest is the inverse without them."""
    torch = pytest.importorskip("torch")
    L = native.load()
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4 * np.sqrt(n) * np.eye(n)
    A = np.stack([a, a])
    A[0, n // 2, n // 3] = np.nan
    A[1, n // 2, n // 2] = np.inf
    dA = torch.from_numpy(np.ascontiguousarray(A.transpose(0, 2, 1))).cuda()
    X = torch.zeros_like(dA)
    info = torch.zeros(2, dtype=torch.int32, device="cuda")
    work = torch.empty(L.negf_b200_zinv_work_bytes(2, n), dtype=torch.uint8, device="cuda")
    assert L.negf_b200_zinv_batched(2, n, _dp(dA), _dp(X), _ip(info), ctypes.c_void_p(work.data_ptr()),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    x = X.cpu().numpy().transpose(0, 2, 1)
    assert np.isnan(x[0]).any()
    keep = np.arange(n) != n // 2
    ref = np.linalg.inv(a[np.ix_(keep, keep)])
    if np.isfinite(x[1]).all():                                    # (n > 64: products with Inf make NaN)
        assert np.abs(x[1][np.ix_(keep, keep)] - ref).max() <= 1e-12
    else:
        assert n > 64


def test_split_calls_match_one_launch(gpu_ctx):
    """Calls with few points run the contacts of all points first, then their
    sweeps (two launches); a workspace limit that leaves no room for the
    contacts' blocks keeps them in one.  The same bits, for devices with
    different numbers of contacts in one call, terminals, dephasing and the
    density matrix with its outer blocks."""
    d2, d3 = G.transport_c0(nbl=4, n=20, seed=5), G.uneven([20, 12, 33, 20], seed=6, cblk=[1, 3, 4])
    d1 = G.transport_c0(nbl=3, n=20, seed=7, cblk=[1])
    hs = [gpu_ctx.upload(d) for d in (d2, d3, d1)]
    ids = np.tile(np.asarray(hs, dtype=np.int32), 5)
    E = np.linspace(-1.2, 1.2, ids.size)
    z, w = np.array([0.1 + 0.3j, -0.4 + 0.1j]), np.array([0.5 + 0.1j, 0.2 - 0.3j])
    frm = np.stack([np.linspace(1, 0, 5), np.linspace(0, 1, 5)], axis=1)

    def solve():
        out = [gpu_ctx.transmission_dos(hs[1], E, eta=1e-3, dos_delta=1e-3),
               gpu_ctx.transmissions(hs[1], E, [(1, 2), (2, 3)], eta=1e-3)]
        mw = gpu_ctx.meir_wingreen(hs[0], E[:5], frm, coupling=0.1, eta=1e-3)
        (d, u, l), (dc, cd), nc, st = gpu_ctx.density_neq(hs[0], E[:1], [1.0], frm[:1], eta=1e-3)
        (rd, ru, rl), (rdc, rcd), rnc, rst = gpu_ctx.density(hs[0], z[:1], w[:1])
        flat = [x for o in out for x in o if x is not None] + [mw[k] for k in sorted(mw)]
        return flat + d + u + l + dc + cd + [nc, st] + rd + ru + rl + rdc + rcd + [rnc, rst]

    try:
        gpu_ctx.set_options(schedule=1, scba_niter=3)
        n0 = gpu_ctx.launch_count()
        a = solve()
        split = gpu_ctx.launch_count() - n0
        # one team's slots of the largest call (the lesser sweeps: 15 + 2 + 8 x 4 + 2 slots of order 33)
        gpu_ctx.set_workspace_limit(256 + 17 * 53 * 33 * 33)
        n0 = gpu_ctx.launch_count()
        b = solve()
        assert gpu_ctx.launch_count() - n0 < split
        assert len(a) == len(b) and all(np.array_equal(x, y) for x, y in zip(a, b))
        gpu_ctx.set_workspace_limit(0)
        # 1, 2 and 3 contacts in one call
        T, dos, nc, st = gpu_ctx.transmission_dos(ids[ids != hs[2]], E[ids != hs[2]], eta=1e-3, dos_delta=1e-3)
        for h in hs[:2]:
            k = ids[ids != hs[2]] == h
            T1, dos1, nc1, st1 = gpu_ctx.transmission_dos(h, E[ids == h], eta=1e-3, dos_delta=1e-3)
            assert np.array_equal(T[k], T1) and np.array_equal(dos[k][:, :dos1.shape[1]], dos1)
            assert np.array_equal(nc[k], nc1) and np.array_equal(st[k], st1)
        T3, dos3, nc3, st3 = gpu_ctx.transmission_dos(hs[2], E, eta=1e-3, dos_delta=1e-3, ni=1, nf=1)
        assert np.all(T3 == 0.0) and np.all(st3 == 0) and np.all(nc3 > 0)
    finally:
        gpu_ctx.set_workspace_limit(0)
        gpu_ctx.set_options()
        for h in hs:
            gpu_ctx.release(h)


@pytest.mark.parametrize("npts", [149, 297])
def test_last_wave_in_a_launch_of_its_own(gpu_ctx, npts):
    """149 points have 298 contacts and 297 points as many sweeps: a little
    over one wave of 296 CTAs, whose rest runs with larger teams.  The same
    bits as in calls that fit one wave."""
    h = gpu_ctx.upload(G.transport_c0(nbl=3, n=84, seed=9))
    E = np.linspace(-1.4, 1.4, npts)
    try:
        n0 = gpu_ctx.launch_count()
        got = gpu_ctx.transmission_dos(h, E, eta=1e-3, dos_delta=1e-3)
        whole = gpu_ctx.launch_count() - n0
        n0 = gpu_ctx.launch_count()
        parts = [gpu_ctx.transmission_dos(h, e, eta=1e-3, dos_delta=1e-3) for e in np.array_split(E, 3)]
        assert whole == 3 and gpu_ctx.launch_count() - n0 == 6
        for k, x in enumerate(got):
            assert np.array_equal(x, np.concatenate([p[k] for p in parts]))
        assert np.all(got[3] == 0)
    finally:
        gpu_ctx.release(h)


@pytest.mark.parametrize("n", [1, 7, 16, 31, 32])
def test_small_orders_by_one_or_two_ctas(gpu_ctx, n):
    """Up to as many points as SMs two CTAs share a point, a contact each; with
    more, one CTA does both.  The same bits, cycle counts and statuses, with a
    non-finite lead on either side and on both."""
    hs = []
    for side in (None, 0, 1, 2):
        dev = G.transport_c0(nbl=3, n=n, seed=11)
        for c in range(2):
            if side in (c, 2):
                dev.lead_h00[c][0, 0] = np.nan
        hs.append(gpu_ctx.upload(dev))
    E = np.linspace(-1.1, 1.1, 160)
    ids = np.asarray(hs, dtype=np.int32)[np.arange(160) % 4]
    try:
        one = gpu_ctx.transmission(ids, E, eta=1e-3, check=False)
        two = [gpu_ctx.transmission(i, e, eta=1e-3, check=False)
               for i, e in zip(np.array_split(ids, 4), np.array_split(E, 4))]
        for k, x in enumerate(one):
            assert np.array_equal(x, np.concatenate([t[k] for t in two]), equal_nan=k == 0)
        good = ids == hs[0]
        assert np.all(one[2][good] == 0) and np.all(one[2][~good] != 0)
    finally:
        for h in hs:
            gpu_ctx.release(h)


@pytest.mark.parametrize("dev", [
    lambda: G.uneven([48, 90, 41, 70], seed=3),
    lambda: G.transport_c1(nbl=3, n=65, seed=2),
], ids=["uneven", "n65_S"])
def test_products_side_by_side(gpu_ctx, dev):
    """Teams run independent products of the sweeps side by side, one CTA one
    after another: the same bits, in the lesser and SCBA sweeps and in the
    density matrix (299 further points of weight zero leave the sum alone)."""
    h = gpu_ctx.upload(dev())
    E = np.linspace(-1.2, 1.2, 300)
    frm = np.stack([np.linspace(1, 0, 300), np.linspace(0, 1, 300)], axis=1)
    z, w = np.full(300, 0.1 + 0.3j), np.zeros(300, dtype=np.complex128)
    w[0] = 0.5 + 0.1j

    def flat(x):
        return [x] if isinstance(x, np.ndarray) else [y for v in x for y in flat(v)]

    try:
        gpu_ctx.set_options(scba_niter=2)
        one = gpu_ctx.meir_wingreen(h, E, frm, coupling=0.1, eta=1e-3)
        rho = flat(gpu_ctx.density(h, z, w)[:2])
        for m in (1, 30, 80):
            team = gpu_ctx.meir_wingreen(h, E[:m], frm[:m], coupling=0.1, eta=1e-3)
            for k in sorted(one):
                assert np.array_equal(team[k], one[k][:m]), k
            part = flat(gpu_ctx.density(h, z[:m], w[:m])[:2])
            assert all(np.array_equal(x, y) for x, y in zip(part, rho))
    finally:
        gpu_ctx.set_options()
        gpu_ctx.release(h)


@pytest.mark.parametrize("n", [20, 48, 100])
def test_decimation_that_is_not_finite_counts_as_not_converged(n):
    """NaN or Inf in a coupling block: max|C1| is not finite, and the count is
    the cap plus one, with a CTA or with a team per problem; the problems
    beside it are not touched."""
    torch = pytest.importorskip("torch")
    L = native.load()
    dev = G.transport_c0(nbl=3, n=n, seed=5)
    z = (0.3 + 1e-3j) * np.eye(n)
    blocks = (z - dev.lead_h00[0], -dev.lead_h01[0], -dev.lead_h01[0].conj().T)
    for batch in (3, 296):
        A, B, C = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda().expand(batch, n, n).contiguous()
                   for x in blocks)
        C[1, n // 2, n // 3] = float("nan")
        B[2, 0, n - 1] = float("inf")
        Go = torch.zeros_like(A)
        nc = torch.zeros(batch, dtype=torch.int32, device="cuda")
        work = torch.empty(L.negf_b200_decimation_work_bytes(batch, n), dtype=torch.uint8, device="cuda")
        assert L.negf_b200_decimation_batched(batch, n, _dp(A), _dp(B), _dp(C), _dp(Go), _ip(nc), 1e-9, 50,
                                              ctypes.c_void_p(work.data_ptr()),
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        k = nc.cpu().numpy()
        assert k[1] == 51 and k[2] == 51
        assert 0 < k[0] < 50 and np.all(np.delete(k, [1, 2]) == k[0])
        assert bool(torch.isfinite(torch.view_as_real(Go[0])).all())


@pytest.mark.parametrize("n", [1, 31, 33, 64])
@pytest.mark.parametrize("dagger", [0, 1, 2])
@pytest.mark.parametrize("place", ["A", "B"])
def test_product_in_the_place_of_an_operand(n, dagger, place):
    """Up to order 64 a product may be written over one of its operands: the
    bits of the product written elsewhere."""
    torch = pytest.importorskip("torch")
    L = native.load()
    g = torch.Generator(device="cuda").manual_seed(n + dagger)
    al, be = (ctypes.c_double * 2)(0.5, -1.0), (ctypes.c_double * 2)(0.25, 0.5)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for batch in (1, 7, 300):
        A, B = (torch.randn((batch, n, n), dtype=torch.complex128, device="cuda", generator=g) for _ in range(2))
        ref = (A if place == "A" else B).clone()
        out = A if place == "A" else B
        for C in (ref, out):
            assert L.negf_b200_zgemm_batched(batch, n, n, n, al, _dp(A), 2 * n * n, _dp(B), 2 * n * n, be, _dp(C),
                                             2 * n * n, dagger, s) == 0
        torch.cuda.synchronize()
        assert torch.equal(out, ref)


def _team_of(L, work, n):
    """The library's own choice of CTAs per matrix (its zinv_shape: two ints in
    one register), so that a test says which sizes it compares."""
    f = L["_ZN4negf10zinv_shapeEiiii"]
    f.restype, f.argtypes = ctypes.c_uint64, [ctypes.c_int] * 4
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return int(f(work, n, 2 * sms, sms) & 0xffffffff)


@pytest.mark.parametrize("n", [64, 65, 96, 127, 129, 256, 257, 512, 513])
def test_inverse_bits_of_one_cta_and_of_teams(n):
    """One wave of matrices (a CTA each) against calls small enough for teams
    of every size the order takes."""
    torch = pytest.importorskip("torch")
    L = native.load()
    batch = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    assert _team_of(L, batch, n) == 1
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((batch, n, n), dtype=torch.complex128, device="cuda", generator=g)
    info = torch.full((batch,), -1, dtype=torch.int32, device="cuda")
    work = torch.empty(L.negf_b200_zinv_work_bytes(batch, n), dtype=torch.uint8, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    w = ctypes.c_void_p(work.data_ptr())
    X = torch.zeros_like(A)
    assert L.negf_b200_zinv_batched(batch, n, _dp(A), _dp(X), _ip(info), w, s) == 0
    assert int(info.abs().max()) == 0
    sizes = {}
    for m in range(batch - 1, 0, -1):
        sizes[_team_of(L, m, n)] = m                               # the fewest matrices of each team size
    sizes.pop(1, None)
    assert max(sizes) >= (4 if n <= 80 else 16)
    for team, m in sizes.items():
        Y = torch.zeros_like(A[:m])
        assert L.negf_b200_zinv_batched(m, n, _dp(A), _dp(Y), _ip(info), w, s) == 0
        torch.cuda.synchronize()
        assert torch.equal(Y, X[:m]), team


@pytest.mark.parametrize("batch", [2, 296])
@pytest.mark.parametrize("n", [65, 100, 200, 300, 600])
def test_inverse_with_an_infinite_pivot_above_one_panel(n, batch):
    """An infinite diagonal entry of a matrix with a dominant diagonal is the
    pivot of its own column, with reciprocal 0: its row and column of the
    inverse vanish and the rest is the inverse without them, to
    8 n u kappa |inv| (LAPACK's own error is within it too)."""
    torch = pytest.importorskip("torch")
    L = native.load()
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 8 * np.sqrt(n) * np.eye(n)
    keep = np.arange(n) != n // 2
    sub = a[np.ix_(keep, keep)]
    ref = np.linalg.inv(sub)
    a[n // 2, n // 2] = np.inf
    dA = torch.from_numpy(np.ascontiguousarray(a.T)).cuda().expand(batch, n, n).contiguous()
    X = torch.zeros_like(dA)
    info = torch.zeros(batch, dtype=torch.int32, device="cuda")
    work = torch.empty(L.negf_b200_zinv_work_bytes(batch, n), dtype=torch.uint8, device="cuda")
    assert L.negf_b200_zinv_batched(batch, n, _dp(dA), _dp(X), _ip(info), ctypes.c_void_p(work.data_ptr()),
                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    x = X[batch - 1].cpu().numpy().T
    assert bool((X == X[0]).all())
    assert np.all(x[n // 2] == 0) and np.all(x[:, n // 2] == 0)
    bound = 16 * n * 2.0 ** -53 * np.linalg.cond(sub) * np.linalg.norm(ref, 2)
    assert np.abs(x[np.ix_(keep, keep)] - ref).max() <= bound
