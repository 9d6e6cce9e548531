"""Second-order optimizers on the GPU: the batched QR of the eigenbasis refresh against Householder QR,
and SOAP trajectories with either of them."""

import pytest
import torch

import heavyball_b200 as hb
from heavyball_b200 import utils
from heavyball_b200.utils.orthogonal import _panel_cholesky_qr

pytestmark = pytest.mark.gpu


def _spd_power_iterate(n, batch, decades, noise, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    basis = torch.linalg.qr(torch.randn(batch, n, n, device="cuda", dtype=torch.float64, generator=gen)).Q
    gg = (basis * torch.logspace(0, -decades, n, device="cuda", dtype=torch.float64)) @ basis.mT
    q_old = torch.linalg.qr(basis + noise * torch.randn(batch, n, n, device="cuda", dtype=torch.float64, generator=gen)).Q
    return (gg @ q_old).float()


@pytest.mark.parametrize("decades,noise", [(2, 1e-2), (10, 1e-3), (20, 1.0)])
def test_panel_qr_is_orthonormal_and_matches_householder(decades, noise):
    power = _spd_power_iterate(512, 4, decades, noise)
    q = _panel_cholesky_qr(power)
    assert q is not None
    eye = torch.eye(512, device="cuda")
    assert (q.mT @ q - eye).abs().max().item() < 1e-5
    if decades == 2:
        ref = torch.linalg.qr(power.double()).Q
        assert ((q.double() * ref).sum(-2).abs() - 1).abs().max().item() < 1e-4


def _train(fast, steps=6):
    torch.manual_seed(0)
    utils.fast_qr = fast
    try:
        ws = [torch.nn.Parameter(torch.randn(128, 96, device="cuda") * 0.1) for _ in range(3)]
        target = [torch.randn_like(w) for w in ws]
        opt = hb.SOAP(ws, lr=1e-2, precondition_frequency=2, warmup_steps=0)
        for _ in range(steps):
            loss = sum(((w @ w.mT @ t - t) ** 2).mean() for w, t in zip(ws, target))
            loss.backward()
            opt.step()
            opt.zero_grad()
        return [w.detach().clone() for w in ws]
    finally:
        utils.fast_qr = True


def test_soap_trajectory_does_not_depend_on_qr_flavour():
    """Column signs of the eigenbasis cancel in the update, so both QR routes give the same parameters."""
    a, b = _train(True), _train(False)
    for x, y in zip(a, b):
        assert torch.isfinite(x).all()
        assert (x - y).abs().max().item() < 2e-3 * y.abs().max().item()


def test_recursive_triangular_solve_matches_library():
    """PSGD's ``V Q^-1``: recursion over column blocks with tensor-core products against cuBLAS TRSM."""
    from heavyball_b200.utils.psgd import _solve_right_upper

    torch.manual_seed(0)
    for d, rows in ((1024, 512), (640, 300), (100, 64)):
        q = torch.randn(4, d, d, device="cuda").triu() * 0.05 + torch.eye(d, device="cuda") * 2
        b = torch.randn(4, rows, d, device="cuda")
        got = _solve_right_upper(q, b)
        ref = torch.linalg.solve_triangular(q.double(), b.double(), upper=True, left=False)
        lib = torch.linalg.solve_triangular(q, b, upper=True, left=False)
        err = (got.double() - ref).abs().max().item()
        lib_err = (lib.double() - ref).abs().max().item()
        assert err < max(20 * lib_err, 1e-4), (d, err, lib_err)
    hb.ops.check_status()


def test_psgd_kron_steps_with_tensor_core_products_match_library_products():
    def run(flag):
        utils.tensor_core_matmul = flag
        try:
            torch.manual_seed(0)
            ws = [torch.nn.Parameter(torch.randn(256, 192, device="cuda") * 0.1) for _ in range(2)]
            opt = hb.PSGDKron(ws, lr=1e-3, preconditioner_update_probability=1.0)
            for _ in range(4):
                torch.manual_seed(1)
                loss = sum((w @ w.mT).square().mean() for w in ws)
                loss.backward()
                opt.step()
                opt.zero_grad()
            return [w.detach().clone() for w in ws]
        finally:
            utils.tensor_core_matmul = True

    a, b = run(True), run(False)
    for x, y in zip(a, b):
        assert torch.isfinite(x).all()
        assert (x - y).abs().max().item() < 1e-3 * y.abs().max().item()


@pytest.mark.parametrize("n,k,m,p", [(1024, 1024, 512, 32), (1000, 300, 7, 32), (130, 64, 64, 32), (4096, 256, 224, 20)])
def test_tall_skinny_products_match_matmul(n, k, m, p):
    ext = hb.ops.load()
    torch.manual_seed(0)
    base = torch.randn(3, n, k, device="cuda")
    w = torch.randn(3, n, p, device="cuda")
    parts = ext.tall_t_mul(base, m, w)
    ref = base[..., :m].double().mT @ w.double()
    assert parts.shape[1:] == (3, m, p)
    assert torch.allclose(parts.sum(0).double(), ref, atol=1e-3, rtol=1e-4)


def test_cholesky_qr2_fast_path_and_its_failure_flag():
    """Well-conditioned refresh inputs take two rounds of Cholesky QR (matrix products only); badly conditioned ones are
    flagged on the device, and ``_qr_basis`` then climbs to the variants with shifted rounds in front (or, past those,
    to the panel-wise method)."""
    from heavyball_b200.utils import orthogonal
    from heavyball_b200.utils.orthogonal import _cholesky_qr2, _qr_basis

    eye = torch.eye(512, device="cuda")
    easy = _spd_power_iterate(512, 4, 2, 1e-2)
    q, bad = _cholesky_qr2(easy)
    assert int(bad.sum()) == 0
    assert (q.mT @ q - eye).abs().max().item() < 3e-5
    ref = torch.linalg.qr(easy.double()).Q
    assert ((q.double() * ref).sum(-2).abs() - 1).abs().max().item() < 1e-4
    hard = _spd_power_iterate(512, 4, 20, 1.0)
    _, bad = _cholesky_qr2(hard)
    assert int(bad.sum()) > 0
    before = dict(orthogonal.qr_stats)
    q = _qr_basis(hard)
    assert (q.mT @ q - eye).abs().max().item() < 1e-4
    assert orthogonal.qr_stats["cholesky_qr2"] == before["cholesky_qr2"]  # the plain variant was refused ...
    assert sum(orthogonal.qr_stats.values()) == sum(before.values()) + 1  # ... and exactly one other route produced it
    for _ in range(3):  # replayed from its graph from the second call on
        q = _qr_basis(easy)
    assert (q.mT @ q - eye).abs().max().item() < 3e-5


@pytest.mark.parametrize("decades,shifted", [(2, 0), (5, 1), (7, 3)])
def test_shifted_cholesky_qr_reaches_worse_conditioning(decades, shifted):
    """Every variant returns the Householder factor's Q (up to column signs) while the input is within its reach."""
    from heavyball_b200.utils.orthogonal import _cholesky_qr2

    torch.manual_seed(decades)
    n = 512
    u = torch.linalg.qr(torch.randn(2, n, n, device="cuda", dtype=torch.float64)).Q
    v = torch.linalg.qr(torch.randn(2, n, n, device="cuda", dtype=torch.float64)).Q
    a = (u * torch.logspace(0, -decades, n, device="cuda", dtype=torch.float64)) @ v.mT
    q, bad = _cholesky_qr2(a.float(), shifted)
    assert int(bad.sum()) == 0
    assert (q.mT @ q - torch.eye(n, device="cuda")).abs().max().item() < 1e-4
    if decades <= 5:  # beyond that the trailing columns of the fp32 input are rounding noise in any method
        ref = torch.linalg.qr(a).Q
        assert ((q.double() * ref).sum(-2).abs() - 1).abs().max().item() < 1e-2


@pytest.mark.parametrize("n", [128, 300, 1024])
def test_blocked_cholesky_with_the_leaf_kernel(n):
    """128-wide leaves are factored and inverted by one kernel for the whole batch; the inverses serve every solve of
    the recursion.  A matrix that is not positive definite is counted, the others are unaffected."""
    from heavyball_b200.utils.orthogonal import _chol_upper_blocked, _leaf_inverse_buffer

    torch.manual_seed(n)
    B = 3
    x = torch.randn(B, n, 2 * n, device="cuda", dtype=torch.float64)
    g64 = x @ x.mT / (2 * n) + 0.1 * torch.eye(n, device="cuda", dtype=torch.float64)
    g = g64.float()
    g[1, n // 2, n // 2] = -1.0  # breaks matrix 1 only
    ref = torch.linalg.cholesky(g64, upper=True)
    work, r = g.clone(), torch.zeros_like(g)
    bad = torch.zeros(B, dtype=torch.int32, device="cuda")
    inv = _leaf_inverse_buffer(work)
    assert inv is not None
    _chol_upper_blocked(work, r, bad, 0, n, inv)
    torch.cuda.synchronize()
    assert bad.tolist()[0] == 0 and bad.tolist()[2] == 0 and bad.tolist()[1] > 0
    for b in (0, 2):
        assert float((r[b].double() - ref[b]).abs().max()) < 2e-4 * float(ref[b].abs().max())
        assert float(r[b].tril(-1).abs().max()) == 0
        for blk in range((n + 127) // 128):
            lo, hi = blk * 128, min(n, blk * 128 + 128)
            want = torch.linalg.inv(r[b, lo:hi, lo:hi].double())
            got = inv[b, blk, : hi - lo, : hi - lo].double()
            assert float((got - want).abs().max()) < 1e-3 * float(want.abs().max())


@pytest.mark.parametrize("n,r", [(5000, 7), (300_000, 23), (1_000_003, 32)])
def test_skinny_gram_of_very_tall_matrices(n, r):
    """``A^T B`` over millions of rows (the low-rank preconditioner's flattened parameter vector) on the long-dimension
    product kernel, cut into enough slices to fill the machine."""
    from heavyball_b200.utils.psgd import _skinny_gram

    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn(n, r, device="cuda", generator=g)
    b = torch.randn(n, r, device="cuda", generator=g)
    got = _skinny_gram(a, b)
    want = a.double().T @ b.double()
    assert got.shape == (r, r)
    assert float((got.double() - want).abs().max()) < 1e-5 * float((a.double().abs().T @ b.double().abs()).max())


@pytest.mark.parametrize("B,n,k", [(2, 1, 1), (3, 9, 257), (2, 260, 1024), (1, 5, 12288), (1, 3, 12289)])
def test_columns_in_order_and_back(B, n, k):
    """Moved as bits, NaN and infinities too; one column past what the kernel takes goes the general way."""
    from heavyball_b200.utils.soap import _permute_columns

    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(B, n, k, device="cuda", generator=g)
    x[0, 0, 0], x[0, -1, -1] = float("nan"), float("-inf")
    order = torch.stack([torch.randperm(k, device="cuda", generator=g) for _ in range(B)])
    moved = _permute_columns(x, order)
    assert torch.equal(moved.view(torch.int32), x.view(torch.int32).gather(-1, order.unsqueeze(-2).expand_as(x)))
    assert torch.equal(_permute_columns(moved, order, inverse=True).view(torch.int32), x.view(torch.int32))


@pytest.mark.parametrize("B", [65535, 65536])
def test_columns_of_more_matrices_than_a_grid_has(B):
    """The kernel counts matrices in the grid's second dimension; one more goes the general way."""
    from heavyball_b200.utils.soap import _permute_columns

    g = torch.Generator(device="cuda").manual_seed(B)
    x, order = torch.randn(B, 2, 3, device="cuda", generator=g), torch.rand(B, 3, device="cuda", generator=g).argsort(-1)
    moved = _permute_columns(x, order)
    assert torch.equal(moved, x.gather(-1, order.unsqueeze(-2).expand_as(x))) and torch.equal(_permute_columns(moved, order, inverse=True), x)


@pytest.mark.parametrize("k", [1, 33, 256, 1000])
def test_identity_defect_flags_what_the_definition_flags(k):
    from heavyball_b200 import ops

    base = torch.eye(k, device="cuda").expand(6, k, k)
    padded = torch.full((6, k, k + 3), 9.0, device="cuda")
    gram = padded[..., :k].copy_(base)
    gram[1, -1, -1] += 2e-4
    gram[2, k // 2, 0] += -2e-4
    gram[3, 0, -1] = float("nan")
    gram[4, -1, 0] = float("inf")
    gram[5] += 0.5e-4
    bad = torch.zeros(6, dtype=torch.int32, device="cuda")
    ops.load().identity_defect(gram, 1e-4, bad)
    assert bad.tolist() == [0, 1, 1, 1, 1, 0]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float64])
@pytest.mark.parametrize("name", ["SOAP", "PSGDKron"])
def test_a_step_does_not_depend_on_the_default_dtype(name, dtype):
    """Scripts that build their models under another default dtype: intermediates of the matrix stages stay fp32."""

    def run(default):
        torch.manual_seed(0)
        ws = [torch.nn.Parameter(torch.randn(200, 333, device="cuda") * 0.1) for _ in range(2)]
        grads = [[torch.randn_like(w) * 1e-2 for w in ws] for _ in range(4)]
        kwargs = dict(preconditioner_update_probability=1.0) if name == "PSGDKron" else dict(precondition_frequency=2)
        opt = getattr(hb, name)(ws, lr=1e-2, **kwargs)
        for i, gs in enumerate(grads):
            for w, g in zip(ws, gs):
                w.grad = g.clone()
            torch.set_default_dtype(default if i == 3 else torch.float32)
            try:
                opt.step()
            finally:
                torch.set_default_dtype(torch.float32)
        return ws

    for got, want in zip(run(dtype), run(torch.float32)):
        assert torch.isfinite(want).all() and float((got - want).abs().max()) < 1e-5 * float(want.abs().max())


@pytest.mark.parametrize("shifted", [0, 1])
@pytest.mark.parametrize("batch,n,k", [(3, 256, 256), (1, 320, 256), (2, 384, 384), (16, 512, 512), (2, 1024, 512), (3, 640, 640), (1, 896, 896), (16, 1024, 1024),
                                       (2, 1152, 1152), (1, 1664, 1664), (2, 2048, 2048)])  # fmt: skip
def test_cholesky_qr_of_whole_blocks_has_the_bits_of_the_block_by_block_form(batch, n, k, shifted, monkeypatch):
    """The chain of ops.chol_qr_round against the same recursion through single products, splits, copies and the library's fp32 product with
    the leaves' inverses: equal bits, and an orthonormal basis, for widths whose halves are even and odd numbers of blocks."""
    from heavyball_b200.utils import orthogonal

    gen = torch.Generator("cuda").manual_seed(k + batch)
    x = torch.eye(n, k, device="cuda") + 0.3 / k**0.5 * torch.randn(batch, n, k, device="cuda", generator=gen)
    x = x * torch.logspace(2, -2, k, device="cuda")
    assert orthogonal._whole_blocks(x)
    before = x.clone()
    q, bad = orthogonal._cholesky_qr2(x, shifted)
    monkeypatch.setattr(orthogonal, "_whole_blocks", lambda a: False)
    want, want_bad = orthogonal._cholesky_qr2(x, shifted)
    assert torch.equal(x, before) and torch.equal(bad, want_bad) and int(bad.sum()) == 0
    assert torch.equal(q, want), float((q - want).abs().max())
    defect = (q.double().mT @ q.double() - torch.eye(k, device="cuda", dtype=torch.float64)).abs().max()
    assert defect < 1e-4


@pytest.mark.parametrize("graph_qr", [True, False])
@pytest.mark.parametrize("start", [1, 2, 3, 4])
def test_basis_of_a_view_that_starts_anywhere(start, graph_qr, monkeypatch):
    """A contiguous view into a flat buffer gives what a matrix of its own gives, on the first, the captured and the replayed call.  The singular
    values lie within 1 +- 0.6: sums in another order move a basis by a few units of 2^-24 times the root of 256, below 1e-5."""
    monkeypatch.setattr(utils, "graph_qr", graph_qr)
    flat = 0.3 / 16 * torch.randn(256 * 256 + start, device="cuda", generator=torch.Generator("cuda").manual_seed(4))
    view = flat[start:].view(256, 256)
    view += torch.eye(256, device="cuda")
    for _ in range(3):
        torch.testing.assert_close(utils.inplace_orthogonal_(view, "qr"), utils.inplace_orthogonal_(view.clone(), "qr"), rtol=0, atol=1e-5)


def test_cholesky_qr_refuses_dependent_columns_either_way(monkeypatch):
    from heavyball_b200.utils import orthogonal

    x = torch.randn(2, 512, 512, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    x[1, :, 300] = x[1, :, 5]
    assert orthogonal._cholesky_qr2(x)[1].gt(0).tolist() == [False, True]
    x[0, 7, 9] = float("nan")
    assert orthogonal._cholesky_qr2(x)[1].gt(0).tolist() == [True, True]
    monkeypatch.setattr(orthogonal, "_whole_blocks", lambda a: False)
    assert orthogonal._cholesky_qr2(x)[1].gt(0).tolist() == [True, True]


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 64, 64), (3, 65, 130), (1, 128, 4), (2, 1000, 333), (8, 1024, 1024), (1, 3, 4096)], ids=str)
def test_passes_over_matrices_have_the_bits_of_the_chains_they_replace(shape):
    """Element-wise passes: every operation rounded once in fp32 in either form, subnormal results kept, so equal bits."""
    from heavyball_b200 import ops
    from heavyball_b200.utils import core, psgd

    gen = torch.Generator("cuda").manual_seed(sum(shape))
    draw = lambda *s: torch.randn(*s, device="cuda", generator=gen) * 10.0 ** torch.randint(-40, 3, s, device="cuda", generator=gen)  # noqa: E731
    x = draw(*shape)
    assert torch.equal(core._transposed(x), x.mT.contiguous()) and core._transposed(x).is_contiguous()
    g, v = draw(*shape), draw(*shape)
    assert torch.equal(ops.load().dampen(g, v, 1e-9, 2.0**-23), g + (1e-9 + 2.0**-23 * g.abs()) * v)
    n = shape[-1] if shape[-1] < 2000 else 7
    a, b, ell = draw(shape[0], n, n), draw(shape[0], n, n), draw(shape[0]).abs() + 1e-30
    want = a + b, (a - b).triu()
    got = psgd._sum_and_upper_difference(a.clone(), b.clone())
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    line = draw(shape[0], n * (n + 1) // 2)
    want = line - psgd.triu_to_line([a])[0][1] / ell.view(-1, 1) * 0.1
    assert psgd._packed_step(line, a, ell, 0.1) and torch.equal(line, want)
    dense = psgd.line_to_triu([((shape[0], n, n), line)])[0]
    rows, cols = torch.triu_indices(n, n, device="cuda")
    assert torch.equal(dense[:, rows, cols], line) and torch.equal(dense, dense.triu())


def test_transposes_on_either_side_of_the_rule():
    from heavyball_b200.utils import core

    for shape in [(65535, 4, 4), (3, 31, 4096), (3, 32, 4096), (2, 28, 28), (7, 32, 32), (2, 1000, 127), (16, 600, 129), (1, 129, 130), (64, 129, 130)]:
        flat = torch.randn(shape[0] * shape[1] * shape[2] + 1, device="cuda")
        for x in (flat[:-1].view(shape), flat[1:].view(shape)):
            assert torch.equal(core._transposed(x), x.mT) and core._transposed(x).is_contiguous()


@pytest.mark.parametrize("shape", [(1, 64 * 65535, 32), (1, 64 * 65535 + 1, 32), (1, (1 << 22) - 1, 33), (1, 32, (1 << 22) - 1)], ids=str)
def test_transposes_of_the_longest_matrices(shape):
    from heavyball_b200.utils import core

    x = torch.arange(shape[1] * shape[2], dtype=torch.int32, device="cuda").view(torch.float32).view(shape)  # (bits that all differ)
    assert torch.equal(core._transposed(x).view(torch.int32), x.view(torch.int32).mT)


@pytest.mark.parametrize("n,k", [(1, 3), (7, 130), (64, 1024), (100, 2048), (5, 5000), (9, 12288), (17, 764), (17, 768), (3, 769), (1, 772)])
def test_columns_permuted_and_put_back(n, k):
    x = torch.randn(3, n, k, device="cuda", generator=torch.Generator("cuda").manual_seed(k))
    order = torch.stack([torch.randperm(k, device="cuda") for _ in range(3)])
    y = utils.soap._permute_columns(x, order)
    assert torch.equal(y, x.gather(-1, order.unsqueeze(-2).expand_as(x)))
    assert torch.equal(utils.soap._permute_columns(y, order, inverse=True), x)


@pytest.mark.parametrize("batch,n", [(3, 130), (16, 1024), (11, 2048), (2, 640)])
def test_column_products_of_transposed_copies_have_the_bits_of_the_plain_ones(batch, n):
    """The order of an eigenbasis hangs on the last bits of these sums."""
    from heavyball_b200.utils import core

    gen = torch.Generator("cuda").manual_seed(n)
    q, p = (torch.randn(batch, n, n, device="cuda", generator=gen) for _ in range(2))
    got = torch.einsum("...ji,...ji->...j", core._transposed(q), core._transposed(p))
    assert torch.equal(got, torch.einsum("...ij,...ij->...j", q, p))


@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_products_of_transposed_views_use_them_where_they_lie(ta, tb):
    from heavyball_b200 import ops

    gen = torch.Generator("cuda").manual_seed(5)
    a, b = torch.randn(2, 256, 384, device="cuda", generator=gen), torch.randn(2, 384, 512, device="cuda", generator=gen)
    a = a.mT.contiguous().mT if ta else a
    b = b.mT.contiguous().mT if tb else b
    for product in (ops.matmul16, ops.matmul3):
        assert torch.equal(product(a, b), product(a.contiguous(), b.contiguous()))
        assert torch.equal(product(a.mT, b.mT, True, True), product(a.contiguous(), b.contiguous()))


def test_cycles_are_not_collected_while_a_graph_is_captured():
    """Destroying a captured graph invalidates any capture under way; a cycle may hold one."""
    import gc

    from heavyball_b200.utils import core

    def cycle_with_a_graph():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            torch.ones(8, device="cuda")
        holder = [graph]
        holder.append(holder)

    gc.collect()
    threshold = gc.get_threshold()
    cycle_with_a_graph()
    fresh = torch.cuda.CUDAGraph()
    try:
        gc.set_threshold(1, 1, 1)
        with core._captured_into(fresh):
            objects = [[i] for i in range(2000)]  # would set off a collection of every generation
            x = torch.ones(8, device="cuda") * 3
    finally:
        gc.set_threshold(*threshold)
    assert gc.isenabled() and len(objects) == 2000
    fresh.replay()
    assert x.tolist() == [3.0] * 8


@pytest.mark.parametrize("shape", [(1, 1), (3, 7), (2, 128, 128), (8, 1000, 33), (2, 524800)], ids=str)
def test_scaled_matrices_have_the_bits_of_the_broadcast(shape):
    from heavyball_b200.utils import core

    gen = torch.Generator("cuda").manual_seed(len(shape))
    x = torch.randn(*shape, device="cuda", generator=gen) * 10.0 ** torch.randint(-38, 3, shape, device="cuda", generator=gen)
    by = torch.randn(shape[0], device="cuda", generator=gen)
    wide = by.view(-1, *[1] * (len(shape) - 1))
    want = x * wide
    core._scale_matrices_(x, by)
    assert torch.equal(x, want)


@pytest.mark.parametrize("batch,rows", [(1, 64), (8, 1024), (3, 4096), (2, 192)])
def test_leaf_solve_has_the_bits_of_the_library_product(batch, rows):
    """Sums over the 128 rows of the inverse in their order, each product fused into its sum, in either kernel."""
    from heavyball_b200 import ops

    gen = torch.Generator("cuda").manual_seed(rows)
    wide = torch.randn(batch, rows, 384, device="cuda", generator=gen)
    inv = torch.randn(batch, 3, 128, 128, device="cuda", generator=gen).triu()
    x = torch.full((batch, rows, 256), 7.0, device="cuda")
    ops.load().leaf_solve(wide[..., 128:256], inv, 1, x[..., 128:])
    assert torch.equal(x[..., 128:], torch.bmm(wide[..., 128:256], inv[:, 1])) and bool((x[..., :128] == 7).all())


@pytest.mark.parametrize("turn", [0.0, 0.03])
def test_moments_are_rotated_by_the_product_whose_time_does_not_hang_on_the_values(turn, monkeypatch):
    """A settled basis turns by an identity, and moments in it are all but diagonal: products of fp16 pairs would compute most of such results a
    second time.  Split tf32 in three products: 2^-18 of the sums of magnitudes each."""
    from heavyball_b200 import ops
    from heavyball_b200.utils import soap

    def refuse(*args, **kw):
        raise AssertionError("a product of fp16 pairs")

    monkeypatch.setattr(ops, "matmul16", refuse)
    gen = torch.Generator("cuda").manual_seed(3)
    draw = lambda *s: torch.randn(*s, device="cuda", dtype=torch.float64, generator=gen)  # noqa: E731
    n, m = 256, 384
    old = [torch.linalg.qr(draw(2, k, k)).Q for k in (n, m)]
    new = [torch.linalg.qr(q + turn * draw(2, *q.shape[1:]) / q.shape[1] ** 0.5).Q.float() for q in old]
    old = [q.float() for q in old]
    state = torch.randn(2, n, m, device="cuda", generator=gen)
    rots = [a.double().mT @ b.double() for a, b in zip(new, old)]
    sizes = [a.double().abs().mT @ b.double().abs() for a, b in zip(new, old)]
    got = state.clone()
    soap._rotate_states(old, new, [got])
    off = (got.double() - rots[0] @ state.double() @ rots[1].mT).abs()
    assert bool((off <= 3 * 2.0**-18 * (sizes[0] @ state.double().abs() @ sizes[1].mT)).all())


def _power_iteration_in_64_bits(a, iterations):
    wide = a.double()
    norms = wide.norm(dim=-1)
    top = norms.amax(-1)
    x = wide[torch.arange(a.shape[0]), norms.argmax(-1)] / top[:, None]
    m = wide / top[:, None, None]
    for _ in range(iterations):
        x = torch.einsum("bij,bj->bi", m, torch.einsum("bij,bj->bi", m, x))
        x = x / x.norm(dim=-1, keepdim=True)
    return (x * torch.einsum("bij,bj->bi", m, torch.einsum("bij,bj->bi", m, x))).sum(-1).sqrt() * top


@pytest.mark.parametrize("n,iterations", [(16, 2), (64, 4), (512, 4)])
def test_power_iteration_is_no_further_from_64_bits_than_its_operations(n, iterations, monkeypatch):
    """Scalings round nothing in the kernel, each division once in the operations: root mean square errors of 144 estimates, a twentieth of which
    is the spread of such a figure."""
    from heavyball_b200.utils import psgd

    gen = torch.Generator("cuda").manual_seed(0)
    fall = torch.logspace(0, -1.5, n, device="cuda")
    kinds = [lambda b: b @ b.mT + torch.eye(n, device="cuda"), lambda b: b @ b.mT, lambda b: (b @ b.mT) * fall.view(-1, 1) * fall]
    mats = torch.cat([kinds[i % 3](torch.randn(8, n, n, device="cuda", generator=gen) / n**0.5) for i in range(18)])
    want = _power_iteration_in_64_bits(mats, iterations)
    error = lambda: float(((psgd.max_eigenvalue_spd(mats, iterations).double() - want) / want).square().mean().sqrt())  # noqa: E731
    kernel = error()
    monkeypatch.setattr(psgd, "_own_pass", lambda *ts: None)
    assert kernel <= 1.1 * error()


@pytest.mark.parametrize("batch,n", [(1, 1), (3, 2), (2, 31), (1, 130), (8, 1024), (2, 1001), (3, 2048), (1, 4097)])
@pytest.mark.parametrize("iterations", [0, 2, 4])
@pytest.mark.parametrize("scale", [1.0, 1e-30, 1e15])
def test_power_iteration_in_one_launch_matches_its_operations_in_64_bits(batch, n, iterations, scale, monkeypatch):
    """Sums of n terms in fp32, in another order than the library's: the estimate is a quotient of such sums, good to n 2^-24 at worst and about
    the square root of that in fact; 1e-5 covers the former up to a few hundred and the latter with room.  Scales whose squares leave fp32 are none
    of the iteration's business (row norms overflow there, as they did): 1e15 and 1e-30 stay inside once divided by the largest norm."""
    from heavyball_b200.utils import psgd

    gen = torch.Generator("cuda").manual_seed(n)
    b = torch.randn(batch, n, n, device="cuda", generator=gen) / n**0.5
    a = (b @ b.mT + torch.eye(n, device="cuda")) * scale
    if scale < 1e-20:
        a = a * 1e12  # squares of 1e-18 are normal numbers
    got = psgd.max_eigenvalue_spd(a, power_iter=iterations)
    assert got.shape == (batch,)
    want = _power_iteration_in_64_bits(a, iterations)
    torch.testing.assert_close(got.double(), want, rtol=1e-5, atol=0)


@pytest.mark.parametrize("batch,n", [(37, 20), (38, 300), (75, 200), (150, 128), (149, 129), (300, 64), (75, 512), (1024, 5), (1025, 5), (1100, 64), (1, 1280),
                                     (1, 1284), (2, 1284), (2, 1024), (2, 1025)])  # fmt: skip
def test_power_iteration_of_many_and_of_few_matrices(batch, n, monkeypatch):
    """Clusters of one to sixteen CTAs, and sizes on either side of where the library's operations are the faster."""
    test_power_iteration_in_one_launch_matches_its_operations_in_64_bits(batch, n, 2, 1.0, monkeypatch)


@pytest.mark.parametrize("block,single", [(1, 512), (512, 1), (3, 40), (40, 3), (30, 32), (600, 88), (88, 600), (0, 639), (638, 0)])
def test_power_iteration_starts_from_the_first_of_equal_rows(block, single):
    """Rows (3, 4), (4, 3) and (5): norms of 5 that are exact, in blocks of eigenvalues 7 and 5 that the iteration does not leave."""
    from heavyball_b200.utils import psgd

    a = torch.zeros(1, 640, 640, device="cuda")
    a[0, block, block] = a[0, block + 1, block + 1] = 3
    a[0, block, block + 1] = a[0, block + 1, block] = 4
    a[0, single, single] = 5
    assert abs(float(psgd.max_eigenvalue_spd(a, power_iter=2)) - (7 if block < single else 5)) < 1e-5


def test_power_iteration_of_zeros_and_of_what_is_not_finite():
    from heavyball_b200.utils import psgd

    a = torch.zeros(3, 64, 64, device="cuda")
    a[1] = torch.eye(64, device="cuda")
    a[2, 3, 5] = float("nan")
    got = psgd.max_eigenvalue_spd(a, power_iter=2)
    assert got[0] == 0 and abs(float(got[1]) - 1) < 1e-6 and bool(got[2].isnan())


@pytest.mark.parametrize("count", [-1, -7])
@pytest.mark.parametrize("name", ["PSGDKron", "PSGDPRO"])
def test_a_negative_number_of_power_iterations_is_none(name, count):
    """``range`` of it is empty; the spectral norms next to it take it as a request for the sketch."""
    from heavyball_b200.utils import psgd

    b = torch.randn(3, 96, 96, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    a = b @ b.mT
    torch.testing.assert_close(psgd.max_eigenvalue_spd(a, count), psgd.max_eigenvalue_spd(a, 0), rtol=1e-5, atol=0)
    p = torch.nn.Parameter(torch.randn(128, 128, device="cuda"))
    opt = getattr(hb, name)([p], lr=1e-3, precond_update_power_iterations=count)
    for _ in range(2):
        p.grad = torch.randn_like(p)
        opt.step()
    assert torch.isfinite(p).all()


def _spd(*shape, seed=5):
    b = torch.randn(*shape, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
    return b @ b.mT


def test_power_iteration_and_noise_under_gradients_and_transforms():
    """Kernels in the place of these expressions read values only: where a gradient or a tangent is wanted, or a transform or a trace looks on, the
    expressions run.  Both are sums and products of a few hundred fp32 values: 1e-4 relative."""
    from torch.autograd import forward_ad
    from torch.fx.experimental.proxy_tensor import make_fx

    from heavyball_b200.utils import psgd

    a = _spd(3, 64, 64)
    eig = lambda m: psgd.max_eigenvalue_spd(m, 2)  # noqa: E731
    close = lambda x, y: torch.testing.assert_close(x, y, rtol=1e-4, atol=1e-4 * float(y.abs().max()))  # noqa: E731
    want = eig(a)
    x = a.clone().requires_grad_()
    (slope,) = torch.autograd.grad(eig(x).sum(), x)
    along = torch.randn_like(a)
    change = (slope * along).sum((-2, -1))
    close(torch.func.jvp(eig, (a,), (along,))[1], change)
    with forward_ad.dual_level():
        close(forward_ad.unpack_dual(eig(forward_ad.make_dual(a, along))).tangent, change)
    close(torch.func.vmap(eig)(torch.stack([a, 2 * a])), torch.stack([want, 2 * want]))
    close(make_fx(eig)(a)(4 * a), 4 * want)
    with torch.no_grad():
        assert torch.equal(eig(x), want)
    g = torch.randn(3, 64, 64, device="cuda").requires_grad_()
    v, damped = psgd.dampen_grad(g, 0.5)
    (slope,) = torch.autograd.grad(damped.sum(), g)
    close(slope, 1 + 2.0**-23 * g.sign() * v)
    noisy = torch.func.vmap(lambda m: psgd.dampen_grad(m, 0.5)[1], randomness="different")(g.detach())
    assert noisy.shape == g.shape


def test_factors_written_in_place_are_seen_by_autograd():
    """A balanced or updated factor counts as written to (by a kernel, too), and what would lose a gradient is refused."""
    from heavyball_b200.utils import psgd

    factors = lambda: [torch.eye(128, device="cuda").repeat(2, 1, 1) * s for s in (1.0, 3.0)]  # noqa: E731
    qs = factors()
    psgd.psgd_balance_Q(qs)
    assert all(q._version > 0 for q in qs)
    qs = factors()
    qs[0].requires_grad_()
    with pytest.raises(RuntimeError):
        psgd.psgd_balance_Q(qs)
    with pytest.raises(RuntimeError):  # no gradient is recorded through the solve: refused, not dropped
        utils.core._solve_right_upper(qs[1], torch.randn(2, 128, 128, device="cuda").requires_grad_())
    with pytest.raises(RuntimeError):
        utils.orthogonal._cholesky_qr2(torch.eye(256, device="cuda").requires_grad_())
    packed = [(tuple(q.shape), psgd.triu_to_line([q])[0][1]) for q in factors()]
    before = [line._version for _, line in packed]
    g = torch.randn(2, 128, 128, device="cuda")
    psgd.psgd_update_precond(g, 0.1, packed, True, 0.9, torch.randn_like(g), [torch.zeros(2, device="cuda") for _ in packed], 0.9, 2)
    assert all(line._version >= b + 2 for (_, line), b in zip(packed, before))
