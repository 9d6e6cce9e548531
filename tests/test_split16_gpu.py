"""fp16-pair operands and products on a B200 against 64-bit products: edges of tiles and K blocks, every epilogue, wide ranges."""

import pytest
import torch

from heavyball_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 128, 256], ids=["tile-auto", "tile-128", "tile-256"])
def tile(request):
    ext = ops.load()
    ext.set_split16_gemm_tile(request.param)
    yield request.param
    ext.set_split16_gemm_tile(0)


def _rand(*shape, seed):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


def _off(got, a, b, want=None, floor=0.0):
    """Largest error in units of its bound: 22 bits of either operand and the dropped product of low parts (4 units of 2^-22), and one
    rounding of the accumulator per 16 of K in the last of three walks plus a few for the first two (2^-23 of |a| |b| each).  Blocks that
    are computed in fp32 stay under it, too: sums of 16 products at a time round 16 + K / 16 times by 2^-24."""
    K = a.shape[-1]
    bound = (a.abs() @ b.abs().mT) * (2.0**-20 + (K / 16 + 4) * 2.0**-23) + floor
    return float(((got.double() - (a @ b.mT if want is None else want)).abs() / bound.clamp_min(1e-300)).max())


EDGES = [(1, 128, 128, 64), (2, 127, 129, 65), (1, 257, 255, 193), (3, 1, 256, 1), (1, 2048, 384, 1000), (2, 300, 1030, 3)]


@pytest.mark.parametrize("B,M,N,K", EDGES)
def test_products_and_both_orientations(B, M, N, K, tile):
    a, b = _rand(B, M, K, seed=1), _rand(B, N, K, seed=2)
    wide = torch.full((B, M, N + 5), -7.0, device="cuda")
    out = wide[..., :N]
    ops.split16_gemm(ops.split16(a)[0], ops.split16(b)[0], out=out)
    assert _off(out, a.double(), b.double()) < 1 and bool((wide[..., N:] == -7.0).all())
    at, bt = (torch.empty(B, K, t.shape[1] + 3, device="cuda")[..., : t.shape[1]].copy_(t.mT) for t in (a, b))  # views, odd row strides
    again = torch.empty(B, M, N, device="cuda")
    ops.split16_gemm(ops.split16(at, False, True)[1], ops.split16(bt, False, True)[1], out=again)
    assert torch.equal(again, out)
    ops.check_status()


@pytest.mark.parametrize("R,C", [(5504, 33), (31, 2500), (256, 1024), (257, 1025), (2304, 64)])
def test_operand_of_either_orientation_holds_the_values(R, C):
    """Rows longer than a warp keeps, strips shared by one to eight blocks and by fewer blocks than rows need; padding is zero."""
    x = _rand(2, R, C, seed=3) * torch.logspace(-6, 6, C, device="cuda") * torch.logspace(8, -8, R, device="cuda")[:, None]
    for op, rows in zip(ops.split16(x, True, True), (x, x.mT)):
        kp, n, K = op.data.shape[2] // 2, *rows.shape[1:]
        hi, lo = op.data[..., :kp].double(), op.data[..., kp:].double() / 2048
        got = (hi + lo) * op.unit[:, :n, None].double()
        top = rows.double().abs().amax(-1, keepdim=True)
        assert float(hi.abs().max()) <= 2**15 and float(hi.abs().amax(-1).min()) >= 2**14
        assert bool(((got[..., :K] - rows.double()).abs() <= torch.maximum(rows.double().abs() * 2.0**-22, top * 2.0**-50)).all())
        assert bool((op.data[..., K:kp] == 0).all()) and bool((op.data[..., kp + K :] == 0).all())


@pytest.mark.parametrize("B,M,N,K", [(2, 200, 136, 160), (1, 520, 264, 70)])
@pytest.mark.parametrize("mode", ["lerp", "add", "adam", "laprop"])
def test_epilogues(mode, B, M, N, K, tile):
    a, b, old = _rand(B, M, K, seed=4), _rand(B, N, K, seed=5), _rand(B, M, N, seed=6)
    x, out = a.double() @ b.double().mT, old.clone()
    pa, pb = ops.split16(a)[0], ops.split16(b)[0]
    if mode in ("lerp", "add"):
        kwargs = dict(mode=ops.EPI_LERP, w=0.25) if mode == "lerp" else dict(mode=ops.EPI_ADD, alpha=-1.0)
        ops.split16_gemm(pa, pb, out=out, **kwargs)
        want = old.double() * 0.75 + 0.25 * x if mode == "lerp" else old.double() - x
        assert float((out.double() - want).abs().max()) < 1e-5 * float((a.abs() @ b.abs().mT).max())
        return
    m, v = _rand(B, M, N, seed=7) * 0.1, _rand(B, M, N, seed=8).abs()
    m64, v64 = m.double(), v.double() * 0.95 + x * x * (1 - 0.95)
    d = v64.sqrt().clamp(min=1e-8)
    m64 = m64 * 0.9 + (x if mode == "adam" else x / d) * (1 - 0.9)
    ops.split16_gemm(pa, pb, mode=ops.EPI_ADAM if mode == "adam" else ops.EPI_LAPROP, b1=0.9, b2c=0.95, eps=1e-8, m=m, v=v, out=out)
    # 0.95 and 0.9 in fp32 (2^-24 each) and the approximate square root and quotient (2 ulp) dominate the product's error
    for got, want in ((m, m64), (v, v64), (out, m64 / d if mode == "adam" else m64)):
        assert float((got.double() - want).abs().max()) < 2e-5 * float(want.abs().max())


@pytest.mark.parametrize("B,n,K", [(2, 129, 64), (1, 520, 200), (3, 256, 512)])
def test_symmetric_and_triangular_products(B, n, K, tile):
    x = _rand(B, n, K, seed=9)
    op, out = ops.split16(x)[0], torch.empty(B, n, n, device="cuda")
    ops.split16_gemm(op, op, out=out)
    assert _off(out, x.double(), x.double()) < 1
    r, s = _rand(B, n, n, seed=10).triu(), _rand(B, n, n, seed=11).triu()
    got = ops.matmul16(r, s, upper_upper=True)
    assert _off(got, r.double(), s.double().mT) < 1 and float(got.tril(-1).abs().max()) == 0
    ops.check_status()


@pytest.mark.parametrize("B,n,K", [(1, 1500, 4100), (2, 1300, 4096), (1, 2048, 4128), (2, 1537, 1025), (6, 1280, 512)])
@pytest.mark.parametrize("mode", ["store", "lerp"])
def test_symmetric_split_tf32_has_the_bits_of_small_tiles(mode, B, n, K):
    """Below 96 large tiles, pairs store their diagonal as 128 x 128 tiles do: ragged edges, one and two waves, every branch of the rule."""
    x, old = _rand(B, n, K, seed=19), _rand(B, n, n, seed=20)
    op, _ = ops.tf32_split(x, True, False)
    kwargs = dict(mode=ops.EPI_LERP, w=0.25) if mode == "lerp" else {}
    results = []
    for forced in (0, 128):
        ops.load().set_tf32_gemm_tile(forced)
        results.append(old.clone())
        ops.tf32_gemm(op, op, K, out=results[-1], **kwargs)
    ops.load().set_tf32_gemm_tile(0)
    ops.check_status()
    assert torch.equal(*results)


@pytest.mark.parametrize("B,n,K,tiles", [(2, 1300, 4096, 2), (2, 1537, 1025, 2), (4, 1536, 256, 2), (4, 1536, 255, 0), (7, 1280, 512, 1)])
def test_updates_of_symmetric_views_by_either_tile_of_split_tf32(B, n, K, tiles):
    """Schur complements: subtracted from a view, the tile that the sizes ask for against 128 x 128 tiles."""
    ext, x, old = ops.load(), _rand(B, n, K, seed=40), _rand(B, n, n, seed=41)
    assert ext.tf32_gemm_tiles(n, n, K, B, True) == tiles
    old, op = old + old.mT, ops.tf32_split(x, True, False)[0]
    results = []
    for forced in (0, 128):
        ext.set_tf32_gemm_tile(forced)
        wide = torch.full((B, n + 4, n + 12), -7.0, device="cuda")
        out = wide[:, 4:, 8 : 8 + n].copy_(old)
        ops.tf32_gemm(op, op, K, mode=ops.EPI_ADD, alpha=-1.0, out=out)
        results.append(out)
        assert bool((wide[:, :4] == -7.0).all() and (wide[..., :8] == -7.0).all() and (wide[..., 8 + n :] == -7.0).all())
    ext.set_tf32_gemm_tile(0)
    ops.check_status()
    # 22 bits of either operand and the dropped product, the accumulator rounded once per 8 of K in each of three walks (2^-23), and the sum with
    # the target; kPairTiles (1) computes what small tiles mirror next to the diagonal, so last bits may differ there
    x64 = x.double() @ x.double().mT
    bound = (x.double().abs() @ x.double().abs().mT) * (2.0**-20 + 3 * K / 8 * 2.0**-23) + (old.double().abs() + x64.abs()) * 2.0**-23
    assert bool(((results[0].double() - (old.double() - x64)).abs() <= bound).all())
    assert torch.equal(*results) if tiles != 1 else bool(((results[0] - results[1]).abs() <= 2 * bound).all())


@pytest.mark.parametrize("B,M,N,K", [(3, 1800, 2100, 130), (1, 5000, 3000, 64), (2, 2300, 2304, 200)])
@pytest.mark.parametrize("mode", ["store", "add", "adam"])
def test_pairs_of_ctas_with_several_tiles_each(mode, B, M, N, K):
    """More 256 x 256 tiles than resident pairs: both accumulators, the ring across tiles, the epilogue under the next main loop."""
    assert B * -(-M // 256) * -(-N // 256) > 148
    a, b, out = _rand(B, M, K, seed=42), _rand(B, N, K, seed=43), _rand(B, M, N, seed=44)
    a[0, 5] *= 1e-12  # one row in units of its own
    pa, pb, old = ops.split16(a)[0], ops.split16(b)[0], out.clone()
    m, v = torch.zeros_like(out), torch.zeros_like(out)
    kwargs = {"store": {}, "add": dict(mode=ops.EPI_ADD, alpha=-1.0), "adam": dict(mode=ops.EPI_ADAM, b1=0.5, b2c=0.5, eps=1e-30, m=m, v=v)}[mode]
    results = []
    for forced in (256, 128):
        ops.load().set_split16_gemm_tile(forced)
        ops.split16_gemm(pa, pb, out=out, **kwargs)
        results.append([t.clone() for t in (out, m, v)])
        out.copy_(old), m.zero_(), v.zero_()
    ops.load().set_split16_gemm_tile(0)
    ops.check_status()
    assert all(torch.equal(x, y) for x, y in zip(*results))  # one accumulator per entry and the same walk over K
    if mode == "store":
        assert _off(results[0][0], a.double(), b.double()) < 1


@pytest.mark.parametrize("B,n,K", [(2, 520, 200), (7, 1300, 130)])
@pytest.mark.parametrize("mode", ["lerp", "add"])
def test_symmetric_updates_of_fp16_pairs(mode, B, n, K, tile):
    """Onto a symmetric target that is a view, upper tiles mirrored; the second size gives a pair of CTAs more than one tile."""
    x, old = _rand(B, n, K, seed=45), _rand(B, n, n, seed=46)
    old, op = old + old.mT, ops.split16(x)[0]
    out = torch.empty(B, n, n + 4, device="cuda")[..., :n].copy_(old)
    kwargs = dict(mode=ops.EPI_LERP, w=0.25) if mode == "lerp" else dict(mode=ops.EPI_ADD, alpha=-1.0)
    ops.split16_gemm(op, op, out=out, **kwargs)
    ops.check_status()
    x64 = x.double() @ x.double().mT
    want = old.double() * 0.75 + 0.25 * x64 if mode == "lerp" else old.double() - x64
    # the product's bound and three roundings in fp32 of values up to |old| + |x|
    bound = (x.double().abs() @ x.double().abs().mT) * (2.0**-20 + (K / 16 + 4) * 2.0**-23) + (old.double().abs() + x64.abs()) * 2.0**-22
    assert bool(((out.double() - want).abs() <= bound).all())


def test_ranges_that_fp16_does_not_have(tile):
    """Rows over sixty decades, rows of zeros, of subnormals and with an infinity or a NaN next to ordinary ones."""
    a, b = _rand(1, 300, 96, seed=12), _rand(1, 140, 96, seed=13)
    a, b = a * torch.logspace(-30, 30, 300, device="cuda")[:, None], b * torch.logspace(6, -6, 140, device="cuda")[:, None]
    a[0, 7], a[0, 8], b[0, 3] = 0.0, 1e-41, 0.0
    # (the epilogues' arithmetic flushes results below 2^-126)
    assert _off(ops.matmul16(a, b, False, True), a.double(), b.double(), floor=2.0**-126) < 1
    a[0, 20, 5], a[0, 21, 6], b[0, 9, 1] = float("nan"), float("inf"), float("-inf")
    got, general = ops.matmul16(a, b, False, True), ops.matmul3(a, b, False, True)
    assert torch.equal(torch.isfinite(got), torch.isfinite(general)) and torch.equal(got.isnan(), general.isnan())


@pytest.mark.parametrize("N", [128, 129, 130, 131])
def test_plain_stores_end_with_the_row(N):
    """Rows of a view that end inside a 16-byte unit: nothing past them is written (bulk stores would fill the unit with zeros)."""
    a, b = _rand(2, 200, 96, seed=17), _rand(2, N, 96, seed=18)
    for product in (lambda out: ops.split16_gemm(ops.split16(a)[0], ops.split16(b)[0], out=out),
                    lambda out: ops.tf32_gemm(ops.tf32_split(a)[0], ops.tf32_split(b)[0], 96, out=out)):  # fmt: skip
        wide = torch.full((2, 200, 136), -7.0, device="cuda")
        product(wide[..., :N])
        assert bool((wide[..., N:] == -7.0).all()) and float((wide[..., :N] - a @ b.mT).abs().max()) < 0.1


def test_refused_operands():
    a, b = ops.split16(_rand(1, 128, 64, seed=14))[0], ops.split16(_rand(1, 128, 128, seed=15))[0]
    with pytest.raises(RuntimeError):
        ops.split16_gemm(a, b, out=torch.empty(1, 128, 128, device="cuda"))  # contraction lengths differ
    with pytest.raises(RuntimeError):
        ops.split16_gemm(a, a, out=torch.empty(1, 128, 100, device="cuda"))
    with pytest.raises(RuntimeError):
        ops.split16(_rand(1, 64, 128, seed=16).mT)


@pytest.mark.parametrize("R,C", [(5504, 33), (31, 2500), (257, 1025), (1, 1)])
def test_values_that_are_short_of_bits_are_counted(R, C):
    x = _rand(2, R, C, seed=35)
    x = torch.where(_rand(2, R, C, seed=36) > 1, x * 1e-12, x) * torch.logspace(-20, 20, R, device="cuda")[:, None]
    x[0, 0], x[1, :, 0] = 0.0, 0.0
    for op, rows in zip(ops.split16(x, True, True), (x, x.mT)):
        n = rows.shape[1]
        short = (rows != 0) & (rows.double().abs() < 2.0**-14 * op.unit[:, :n, None].double())
        assert torch.equal(op.short[:, :n].long(), short.sum(-1))


def _graded(B, rows, K, how, seed):
    """Operands whose rows hold values that differ by more than a pair of fp16 numbers covers, opposite zeros of the other operand."""
    a, b = _rand(B, rows, K, seed=seed), _rand(B, K, K, seed=seed + 1)
    h = K // 3
    if how == "identity":  # the result is the graded matrix itself
        return a * torch.logspace(0, -30, K, device="cuda"), torch.eye(K, device="cuda").expand(B, K, K).contiguous()
    a[..., h:] *= float(how)
    b[:, :h, h:], b[:, h:, :h] = 0, 0
    return a, b


@pytest.mark.parametrize("how", ["identity", "1e-9", "1e-12", "1e-15", "1e-30"])
@pytest.mark.parametrize("B,M,K", [(2, 200, 136), (1, 300, 517)])
def test_small_values_opposite_zeros(B, M, K, how, tile):
    """Entry by entry as exact as |a| |b| asks, whichever operand is graded, from rows, columns and views."""
    a, b = _graded(B, M, K, how, 21)
    want = a.double() @ b.double().mT
    pa, pb = ops.split16(a)[0], ops.split16(b)[0]
    out = torch.empty(B, M, K, device="cuda")
    ops.split16_gemm(pa, pb, out=out)
    assert _off(out, a.double(), b.double()) < 1
    turned = torch.empty(B, K, M, device="cuda")
    ops.split16_gemm(pb, pa, out=turned)
    assert _off(turned, b.double(), a.double()) < 1
    at, bt = (torch.empty(B, K, t.shape[1] + 3, device="cuda")[..., : t.shape[1]].copy_(t.mT) for t in (a, b))
    ops.split16_gemm(ops.split16(at, False, True)[1], ops.split16(bt, False, True)[1], out=out)
    assert _off(out, a.double(), b.double()) < 1
    old = _rand(B, M, K, seed=23) * want.abs().float()
    out = old.clone()
    ops.split16_gemm(pa, pb, mode=ops.EPI_LERP, w=0.25, out=out)
    want_lerp = old.double() * 0.75 + 0.25 * want  # in fp32: four roundings of values up to |old| + |x|
    assert bool(((out.double() - want_lerp).abs() <= (old.double().abs() + a.double().abs() @ b.double().abs().mT) * 2.0**-15).all())
    m, v = torch.zeros(B, M, K, device="cuda"), torch.zeros(B, M, K, device="cuda")
    ops.split16_gemm(pa, pb, mode=ops.EPI_ADAM, b1=0.5, b2c=0.5, eps=1e-30, m=m, v=v, out=out)
    assert _off(m, a.double(), b.double(), want * 0.5) < 1
    ops.check_status()


def test_small_values_in_symmetric_and_triangular_products(tile):
    x = _rand(2, 390, 200, seed=24)
    x[:, 130:, :100], x[:, :130, 100:] = 0, 0
    x[:, 130:] *= torch.logspace(0, -16, 100, device="cuda").repeat(2)
    x[:, 131, 100:] *= 1e12
    op, out = ops.split16(x)[0], torch.empty(2, 390, 390, device="cuda")
    ops.split16_gemm(op, op, out=out)
    assert _off(out, x.double(), x.double()) < 1
    r, s = _rand(2, 390, 390, seed=25).triu(), _rand(2, 390, 390, seed=26).triu()
    r, s = r * torch.logspace(0, -15, 390, device="cuda"), s * torch.logspace(0, 15, 390, device="cuda")[:, None]
    s[:, :, 200:] *= 1e-20
    got = ops.matmul16(r, s, upper_upper=True)
    assert _off(got, r.double(), s.double().mT) < 1 and float(got.tril(-1).abs().max()) == 0
    ops.check_status()


def test_values_below_the_normal_range_count(tile):
    """Split tf32 multiplies subnormal values; rows of them, and rows whose only larger values meet zeros."""
    a, b = torch.zeros(1, 130, 140, device="cuda"), _rand(1, 150, 140, seed=27) * 1e20
    a[0, :65] = _rand(65, 140, seed=28) * 1e-41
    a[0, 65:, :70], a[0, 65:, 70:] = 3e-40, 1e-30
    b[0, :, 70:] = 0
    assert _off(ops.matmul16(a, b, False, True), a.double(), b.double()) < 1


def test_sources_are_read_only_where_a_result_hangs_on_them(tile):
    a, b = _rand(2, 300, 256, seed=29), _rand(2, 260, 256, seed=30)
    a[0, 7, 3], b[1, 100, 200] = 1e-12, -1e-30  # short of bits, but lost in sums over ordinary values
    pa, pb, out = ops.split16(a)[0], ops.split16(b)[0], torch.empty(2, 300, 260, device="cuda")
    assert int(pa.short[0, 7]) == 1 and int(pb.short[1, 100]) == 1
    pa.x, pb.x = torch.full_like(a, float("nan")), torch.full_like(b, float("nan"))
    ops.split16_gemm(pa, pb, out=out)
    assert _off(out, a.double(), b.double()) < 1
    with pytest.raises(RuntimeError):  # an output over a source
        ops.split16_gemm(ops.split16(c := _rand(1, 256, 128, seed=33))[0], ops.split16(_rand(1, 128, 128, seed=34))[0], out=c)


@pytest.mark.parametrize("decades", [0, 12, 25])
def test_solves_with_graded_factors_lose_nothing_to_split_tf32(decades):
    """The blocked solve of a preconditioner fit: residual per entry in units of ``|x| |q|``, next to the split-tf32 product's."""
    from heavyball_b200.utils.core import _solve_right_upper

    d, rows = 640, 300
    scale = torch.logspace(0, -decades, d, device="cuda")
    q = (_rand(2, d, d, seed=31).triu(1) * 0.02 + torch.eye(d, device="cuda") * 2) * scale[:, None]
    q[:, :256, 384:] = 0
    b = _rand(2, rows, d, seed=32) * scale.flip(0)

    def residual(pairs):
        x = _solve_right_upper(q, b, pairs=pairs).double()
        return float(((x @ q.double() - b.double()).abs() / (x.abs() @ q.double().abs() + b.double().abs())).max())

    assert residual(True) <= 2 * residual(False) + 2.0**-20


@pytest.mark.parametrize("M,N,K,tb", [(200, 136, 160, False), (129, 300, 130, True), (390, 390, 128, "same")])
def test_accumulation_into_a_view_with_one_allocation(M, N, K, tb, tile):
    """``c -= a op(b)`` on views; the operands of a product share one block of memory (captured regions pay for each of their own)."""
    wide = _rand(2, M, N + 12, seed=37)
    a = _rand(2, M, K + 4, seed=38)[..., :K]
    b = a if tb == "same" else (_rand(2, N, K + 8, seed=39)[..., 8:] if tb else _rand(2, K, N + 4, seed=39)[..., :N])
    c = wide[..., 8 : 8 + N]
    if tb == "same":  # a symmetric product goes onto a symmetric target: upper tiles, mirrored
        c.copy_(c + c.mT.clone())
    old = wide.clone()
    ops.split16_accumulate(c, a, b, bool(tb), -1.0)
    bt = b.double() if tb else b.double().mT
    x = a.double() @ bt.mT
    bound = a.double().abs() @ bt.abs().mT * (2.0**-20 + (K / 16 + 4) * 2.0**-23) + (old[..., 8 : 8 + N].double().abs() + x.abs()) * 2.0**-24
    assert bool(((c.double() - (old[..., 8 : 8 + N].double() - x)).abs() <= bound).all())
    assert torch.equal(wide[..., :8], old[..., :8]) and torch.equal(wide[..., 8 + N :], old[..., 8 + N :])
    count = lambda: torch.cuda.memory_stats()["allocation.all.allocated"]  # noqa: E731
    before = count()
    ops.split16_accumulate(c, a, b, bool(tb), -1.0)
    assert count() - before == 1
    ac, bc = a.contiguous(), b.contiguous()
    before = count()
    ops.matmul16(ac, bc, False, bool(tb))
    assert count() - before == 2
    with pytest.raises(RuntimeError):
        ops.split16_accumulate(ac, ac, bc, bool(tb))
    ops.check_status()


@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("B,M,K,N", [(1, 1, 1, 1), (2, 33, 64, 31), (3, 128, 300, 129), (1, 257, 2100, 40), (2, 1030, 128, 1100)])
def test_operands_of_a_product_from_one_launch(ta, tb, B, M, K, N):
    """The launch that makes both operands of a product gives each what a launch of its own gives (the same bits), whatever cluster the other
    one needs; rows with values too small for 22 bits among them."""
    a, b = _rand(B, *((K, M) if ta else (M, K)), seed=41), _rand(B, *((N, K) if tb else (K, N)), seed=42)
    a[:, ::3] *= 2.0**-20
    b[..., ::5] *= 2.0**-31
    pa = ops.split16(a, not ta, ta)[1 if ta else 0]
    pb = ops.split16(b, tb, not tb)[0 if tb else 1]
    want = torch.empty(B, M, (N + 3) // 4 * 4, device="cuda")[..., :N]
    ops.split16_gemm(pa, pb, out=want)
    assert torch.equal(ops.matmul16(a, b, ta, tb), want)
