"""Edges of tiles, chunks and leaves of the sm_100a kernels: remainders, smallest and largest sizes of a range, several sizes in
one launch.  Oracles are fp64 restatements or the package's PyTorch definitions."""

import pytest
import torch

import heavyball_b200 as hb
from heavyball_b200 import lowering, ops, utils

pytestmark = pytest.mark.gpu
DEV = "cuda"


# ---------------------------------------------------------------------------------------- fused chain


@pytest.mark.parametrize("extra", [(1,), (8_500_000,)], ids=["25 tensors", "more than 8 M elements"])
@pytest.mark.parametrize("ecc", [None, "bf16+8"])
def test_table_in_the_arguments_and_in_memory(ecc, extra):
    """24 small tensors take their table in the launch's arguments; with one more tensor or with too many elements it is in memory:
    the results of the 24 are the same bits either way (rounding noise is addressed by tensor and element)."""
    sizes = [1, 2048, 2049, *range(3, 24)]

    def run(sizes):
        draw = lambda salt: [torch.randn(n, device=DEV, generator=torch.Generator(DEV).manual_seed(100 * salt + i)) for i, n in enumerate(sizes)]  # noqa: E731
        p, g, dtype = draw(1), draw(2), torch.bfloat16 if ecc else torch.float32
        m, v = [t.to(dtype) for t in draw(3)], [t.square().to(dtype) for t in draw(4)]
        residuals = lambda: [torch.zeros(n, dtype=torch.int8, device=DEV) for n in sizes] if ecc else []  # noqa: E731
        me, ve = residuals(), residuals()
        for seed in (5, 6):
            ops.fused_chain(p=p, g=g, s0=m, s0e=me, s1=v, s1e=ve, algo=ops.ADAM, n_state=2, out_mode=ops.OUT_PARAM, dt_p=ops.F32, dt_g=ops.F32,
                            dt_s=ops.BF16E8 if ecc else ops.F32, lr=1e-2, wd=0.1, eps=1e-8, b1=0.9, b2=0.99, seed=seed)  # fmt: skip
        return [t for lst in zip(*[x for x in (p, m, v, me, ve) if x]) for t in lst]

    assert len(sizes) == 24
    for few, more in zip(run(sizes), run([*sizes, *extra])):
        assert torch.equal(few, more)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("sizes", [(1, 3, 4, 1023, 1024, 1025, 4097), (2_500_001, 8193, 7)], ids=len)
@pytest.mark.parametrize("algo,mars,grad,param,count", [
    (ops.ADAM, True, "f32", None, True), (ops.ADAM, False, "f32", None, True), (ops.ADAM, False, "f32", "f32", False),
    (ops.ADAM, False, "bf16", "ecc", False), (ops.EXP_AVG, False, "f32", None, False), (ops.NESTEROV_EMA, False, "f32", None, False),
    (ops.NESTEROV_EMA, True, "bf16", None, False)])  # fmt: skip
def test_rules_known_at_compile_time_match_the_general_kernel(algo, mars, grad, param, count, sizes, shift):
    """Error-corrected state through the instances with the rule compiled in (next vector fetched ahead, random bits drawn before the values
    arrive) and through the general kernel, which a gradient given as the sum over one source selects, over aligned and misaligned starts,
    remainders, zeros and values whose residuals take the slow codec.  The compiler may contract a product and a sum in one of the two:
    2^-24 of a value, which is 2^-8 of a residual's unit (half a unit in the last place of bf16 over 127: 2^-15 of the value), so up to 2^-8 of the
    residuals may come out one unit apart (255 apart where the rounded value goes the other way).  After one launch, whose inputs are the same, no
    pair may stand for a value further off than two units and a few roundings of the terms it was summed from; fp32 results of the second
    differ by a few such roundings and units."""

    def run(extra):
        gen, dtypes = torch.Generator(DEV).manual_seed(3), {"f32": torch.float32, "bf16": torch.bfloat16, "ecc": torch.bfloat16}

        def made(dtype, spread=0.0, positive=False):
            out = []
            for n in sizes:
                x = torch.randn(n, device=DEV, generator=gen) * 10 ** (-spread * torch.rand(n, device=DEV, generator=gen))
                x = torch.where(torch.rand(n, device=DEV, generator=gen) < 0.05, 0.0, x)
                out.append(torch.zeros(n + shift, dtype=dtype, device=DEV)[shift:].copy_(x.abs() if positive else x))
            return out

        residuals = lambda: [t.zero_() for t in made(torch.int8)]  # noqa: E731
        lists = {"g": made(dtypes[grad], 8.0), "s0": made(torch.bfloat16, 35.0), "s0e": residuals()}
        cfg = dict(algo=algo, n_state=1, dt_g=ops.F32 if grad == "f32" else ops.BF16, dt_s=ops.BF16E8, dt_u=ops.F32, b1=0.9, b2=0.99, eps=1e-8)
        if algo == ops.ADAM:
            lists.update(s1=made(torch.bfloat16, 35.0, True), s1e=residuals())
            cfg["n_state"] = 2
        if mars:
            lists.update(mars=made(torch.bfloat16, 35.0), marse=residuals())
            cfg["mars_a"] = -0.0023
        if param is None:
            lists["u"] = made(torch.float32)
            cfg["out_mode"] = ops.OUT_UPDATE
        else:
            lists.update(p=made(dtypes[param]), **({"pe": residuals()} if param == "ecc" else {}))
            cfg.update(out_mode=ops.OUT_PARAM, dt_p=ops.F32 if param == "f32" else ops.BF16E8, lr=1e-2, wd=0.1)
        masked = torch.zeros(len(sizes), dtype=torch.int32, device=DEV)
        if count:
            cfg.update(count_caution=1, masked=masked)
        seen = [{k: [t.clone() for t in v] for k, v in lists.items()}]
        for seed in (5, 6):
            ops.fused_chain(**lists, **cfg, **extra, seed=seed)
            seen.append({k: [t.clone() for t in v] for k, v in {**lists, "masked": [masked]}.items()})
        return seen

    def value(of, name, i):
        x = of[name][i]
        return (utils._ULPState(of[name + "e"][i], 127).decode(x) if name + "e" in of else x).double()

    (before, first, last), (_, first_general, last_general) = run({}), run({"g_delta": [0], "g_scale": 1.0})
    for i in range(len(sizes)):
        g = value(before, "g", i).abs() + (value(before, "mars", i).abs() if mars else 0)
        terms = {"mars": 0 * g, "s0": value(before, "s0", i).abs() + g}
        if algo == ops.ADAM:
            terms["s1"] = value(before, "s1", i) + g * g
            if param is not None:
                terms["p"] = value(before, "p", i).abs() + 1e-2 * terms["s0"] / value(first, "s1", i).sqrt().clamp(min=1e-8)
        for name, scale in terms.items():
            if name in first:
                a, b = value(first, name, i), value(first_general, name, i)
                off = (a - b).abs() - (2.0**-14 * torch.maximum(a.abs(), b.abs()) + 2.0**-21 * scale + 2.0**-133)
                assert bool((off <= 0).all()), (name, i, int(off.argmax()), float(off.max()))
    for name, tensors in last.items():
        for i, (a, b) in enumerate(zip(tensors, last_general[name])):
            if a.dtype in (torch.int8, torch.bfloat16):
                assert int((a != b).sum()) <= a.numel() >> 8, (name, i, int((a != b).sum()))
            else:
                torch.testing.assert_close(a, b, rtol=2**-14, atol=1e-30)


@pytest.mark.parametrize("kind", ["momentum", "momentum-ecc", "caution", "update-ecc", "adam", "adam-bf16", "adam-update",
                                  "adam-ecc", "adam-ecc-param", "adam-ecc-count", "adam-ecc-count-mars"])  # fmt: skip
@pytest.mark.parametrize("sizes", [(1, 3, 4, 5), (1023, 1024, 1025, 4092, 4095), (4096, 4097, 4100, 8188, 8192), (2_000_003, 2_500_000)], ids=str)
def test_whole_and_element_loads_read_the_same_values(sizes, kind):
    """A batch of vectors is loaded whole where all its elements are there and the buffers start on a 16-byte boundary, else
    element by element.  The arithmetic and the random bits of an element don't depend on that: off the boundary the same bits come out."""

    def run(shift):
        gen = torch.Generator(DEV).manual_seed(7)

        def made(dtype, positive=False):
            values = [torch.randn(n, device=DEV, generator=gen) for n in sizes]
            return [torch.zeros(v.numel() + shift, dtype=dtype, device=DEV)[shift:].copy_(v.abs() if positive else v) for v in values]

        masked = torch.zeros(len(sizes), dtype=torch.int32, device=DEV)
        if kind.startswith("momentum"):
            ecc = kind == "momentum-ecc"
            lists = {"g": made(torch.bfloat16 if ecc else torch.float32), "s0": made(torch.bfloat16 if ecc else torch.float32), "u": made(torch.float32)}
            if ecc:
                lists["s0e"] = made(torch.int8)
            cfg = dict(algo=ops.NESTEROV_EMA, n_state=1, b1=0.9, out_mode=ops.OUT_UPDATE, dt_u=ops.F32, dt_p=ops.NONE,
                       dt_g=ops.BF16 if ecc else ops.F32, dt_s=ops.BF16E8 if ecc else ops.F32)  # fmt: skip
        elif kind == "caution":
            lists = {"g": made(torch.bfloat16), "u": made(torch.float32)}
            cfg = dict(algo=ops.IDENTITY, u_is_input=1, count_caution=1, masked=masked, out_mode=ops.OUT_UPDATE,
                       dt_u=ops.F32, dt_g=ops.BF16, dt_s=ops.NONE, dt_p=ops.NONE)  # fmt: skip
        elif kind == "update-ecc":
            lists = {"p": made(torch.bfloat16), "pe": made(torch.int8), "u": made(torch.float32)}
            cfg = dict(algo=ops.IDENTITY, u_is_input=1, out_mode=ops.OUT_PARAM, dt_u=ops.F32, dt_p=ops.BF16E8,
                       dt_g=ops.NONE, dt_s=ops.NONE, lr=1e-2, wd=0.1)  # fmt: skip
        elif kind == "adam-update":
            lists = {"g": made(torch.float32), "s0": made(torch.float32), "s1": made(torch.float32, True), "u": made(torch.float32)}
            cfg = dict(algo=ops.ADAM, n_state=2, b1=0.9, b2=0.99, eps=1e-8, out_mode=ops.OUT_UPDATE, dt_u=ops.F32, dt_p=ops.NONE, dt_g=ops.F32, dt_s=ops.F32)
        elif kind.startswith("adam-ecc"):
            pe, count = kind.endswith("param"), "count" in kind
            g, made8 = made(torch.bfloat16 if pe else torch.float32), lambda: made(torch.int8)
            lists = {"g": g, "s0": made(torch.bfloat16), "s0e": made8(), "s1": made(torch.bfloat16, True), "s1e": made8()}
            if kind.endswith("mars"):
                lists.update(mars=made(torch.bfloat16), marse=made8())
            lists.update({"u": made(torch.float32)} if count else {"p": made(g[0].dtype), **({"pe": made8()} if pe else {})})
            cfg = dict(algo=ops.ADAM, n_state=2, b1=0.9, b2=0.99, eps=1e-8, mars_a=-0.0023, dt_g=ops.BF16 if pe else ops.F32, dt_s=ops.BF16E8)
            cfg.update(dict(out_mode=ops.OUT_UPDATE, dt_u=ops.F32, dt_p=ops.NONE, count_caution=1, masked=masked) if count else
                       dict(out_mode=ops.OUT_PARAM, dt_p=ops.BF16E8 if pe else ops.F32, lr=1e-2, wd=0.1))  # fmt: skip
        else:
            dtype, dt = (torch.float32, ops.F32) if kind == "adam" else (torch.bfloat16, ops.BF16)
            lists = {"p": made(dtype), "g": made(dtype), "s0": made(torch.float32), "s1": made(torch.float32, True)}
            cfg = dict(algo=ops.ADAM, n_state=2, b1=0.9, b2=0.99, eps=1e-8, out_mode=ops.OUT_PARAM, dt_p=dt, dt_g=dt, dt_s=ops.F32, lr=1e-2, wd=0.1)
        ops.fused_chain(**lists, **cfg, seed=3)
        return {**lists, "masked": [masked]}

    whole, elements = run(0), run(1)
    for name, tensors in whole.items():
        for a, b in zip(tensors, elements[name]):
            assert torch.equal(a, b), (name, a.numel(), int((a != b).sum()))


@pytest.mark.parametrize("kw", [{}, {"ecc": "bf16+8", "mars": True, "caution": True}, {"ecc": "bf16+8"}, {"caution": True}], ids=str)
@pytest.mark.parametrize("sizes", [(1,), (2047, 2048, 2049), (8191, 8193, 3, 16384), tuple(range(1, 41)), (10_000_000, 5),
                                   (4095, 4096, 4097, 2_500_001, 7), (8191, 8192, 8193, 1, 10_000_000, 5)], ids=len)  # fmt: skip
def test_fused_chain_at_chunk_edges(sizes, kw):
    """Sizes around the three chunk sizes in launches of the size that takes each (2048 up to 0.9 M or 2.4 M elements, 8192 from
    4.8 M or 9.7 M), more tensors than a warp tests at once, and a launch large enough for the large chunk.
    fp32: a handful of roundings per step (1e-6 of the value); error-corrected state keeps 16 + 8 bits (2^-15 of the value)
    and moves a weight by lr = 1e-2 per step."""
    results = []
    for lowered in (True, False):
        torch.manual_seed(0)
        gen = torch.Generator(DEV).manual_seed(1)
        params = [torch.nn.Parameter(torch.randn(n, device=DEV, generator=gen)) for n in sizes]
        opt = hb.AdamW(params, lr=1e-2, weight_decay=0.1, **kw)
        old, lowering.enabled = lowering.enabled, lowered
        try:
            for _ in range(3):
                for p in params:
                    p.grad = torch.randn(p.shape, device=DEV, generator=gen)
                opt.step()
        finally:
            lowering.enabled = old
        results.append([p.detach() for p in params])
    for a, b in zip(*results):
        # a value next to zero may round to the other side of caution's sign test when its state is stored in fewer bits
        close = torch.isclose(a, b, rtol=1e-5, atol=2e-6 if not kw.get("ecc") else 2e-4)
        assert close.float().mean().item() > (0.999 if kw.get("caution") and a.numel() > 1000 else 1 - 1e-9), (a - b).abs().max()


def _ecc_step(g, prim, res, b1, shift):
    """One momentum step (``s <- s b1 + g``) on error-corrected state; returns what it hands on and the stored pair.  ``shift``:
    elements by which every buffer starts past a 16-byte boundary."""
    place = lambda t: torch.cat([t[:1].expand(shift), t])[shift:] if shift else t.clone()  # noqa: E731
    g, prim, res, out = place(g), place(prim), place(res), place(torch.zeros_like(g))
    ops.fused_chain(g=[g], u=[out], s0=[prim], s0e=[res], algo=ops.HEAVYBALL, n_state=1, b1=b1, seed=11,
                    out_mode=ops.OUT_UPDATE, dt_g=ops.F32, dt_u=ops.F32, dt_s=ops.BF16E8, dt_p=ops.NONE)  # fmt: skip
    return out, prim, res


def _ecc_value(prim, res):
    """The pair's value in 64 bits, and its unit: half a unit in the last place of the primary, over 127."""
    e = torch.where(prim == 0, -126, torch.clamp(torch.frexp(prim.double())[1] - 1, min=-126)).double()
    unit = 2.0 ** (e - 8) / 127
    return prim.double() + res.double() * unit, unit


_FLUSH = 2.0**-126  # single-precision subnormals count as zero in these kernels


@pytest.mark.parametrize("shift", [0, 1], ids=["four at a time", "one at a time"])
def test_ecc_codec_decodes_every_primary(shift):
    """All 65536 primaries (zeros, subnormals, infinities and NaN among them) under random residuals: the value handed on is the
    pair's to fp32 rounding, and the pair that is stored for it again is within one residual unit of it."""
    prim = torch.arange(-32768, 32768, device=DEV, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    prim = prim[torch.randperm(65536, generator=torch.Generator().manual_seed(1)).to(DEV)]
    res = torch.randint(-127, 128, prim.shape, device=DEV, dtype=torch.int8, generator=torch.Generator(DEV).manual_seed(2))
    out, new, left = _ecc_step(torch.zeros(65536, device=DEV), prim, res, 1.0, shift)
    finite = torch.isfinite(prim)
    want, unit = _ecc_value(prim, res)
    assert ((out.double() - want).abs() <= want.abs() * 1e-6 + _FLUSH)[finite].all()
    again, _ = _ecc_value(new, left)
    held = finite & torch.isfinite(new)  # the largest value plus its residual rounds up to infinity
    assert (finite & ~held).sum().item() <= 2
    assert ((again - out.double()).abs() <= unit * 1.001 + 2 * _FLUSH)[held].all()
    assert torch.equal(torch.isnan(out), torch.isnan(prim)) and torch.equal(torch.isnan(new), torch.isnan(prim))
    assert torch.equal(out[torch.isinf(prim)], prim[torch.isinf(prim)].float()) and torch.equal(new[torch.isinf(prim)], prim[torch.isinf(prim)])


def test_ecc_codec_encodes_the_same_bits_four_and_one_at_a_time():
    """fp32 values of all exponents, ties of the bf16 rounding, the largest ones, infinities and NaN.  The primary is the value
    rounded to nearest, the pair is within one residual unit of it, and the codec that handles four values at once stores the
    same bits as the element-wise one (which buffers off a 16-byte boundary take)."""
    gen = torch.Generator(DEV).manual_seed(3)
    bits = torch.randint(-(2**31), 2**31, (1 << 17,), device=DEV, generator=gen)
    ties = (torch.arange(0, 65536, 7, device=DEV) << 16 | 0x8000) - 2**31
    edge = torch.tensor([0x7F7F0000, 0x7F7F7FFF, 0x7F7F8000, 0x7F800000, 0x7FC00000, 0x00800000, 0x007FFFFF, 1, 0, 0x0FFFFFFF, 0x10000000], device=DEV)
    x = torch.cat([bits, ties, edge, edge - 2**31]).to(torch.int32).view(torch.float32)
    zero, none = torch.zeros(x.shape, device=DEV, dtype=torch.bfloat16), torch.zeros(x.shape, device=DEV, dtype=torch.int8)
    out, prim, res = _ecc_step(x, zero, none, 0.0, 0)
    one_out, one_prim, one_res = _ecc_step(x, zero, none, 0.0, 1)
    number = ~torch.isnan(x)
    assert torch.equal(torch.isnan(prim), ~number) and torch.equal(torch.isnan(one_prim), ~number)
    assert torch.equal(out[number], one_out[number])
    assert torch.equal(prim.view(torch.int16)[number], one_prim.view(torch.int16)[number]) and torch.equal(res[number], one_res[number])
    normal = number & (x.abs() >= _FLUSH)
    assert torch.equal(prim[normal], x.to(torch.bfloat16)[normal])
    value, unit = _ecc_value(prim, res)
    held = torch.isfinite(prim) & number
    assert ((value - x.double()).abs() <= unit * 1.001 + 2 * _FLUSH)[held].all()
    assert res[held].to(torch.int32).abs().max().item() <= 127


# ---------------------------------------------------------------------------------------- Newton-Schulz products


def _poly_oracle(x, a, b, c):
    """One polynomial step in fp64 with the kernel's bf16 roundings of S and of the polynomial."""
    s = (x @ x.mT).to(torch.bfloat16).double()
    y = (c * (s @ s) + b * s + a * torch.eye(x.shape[-2], dtype=torch.float64, device=x.device)).to(torch.bfloat16).double()
    return (y @ x).to(torch.bfloat16).double()


@pytest.mark.parametrize("tile", [0, 128, 256])
@pytest.mark.parametrize("shapes", [((64, 64),), ((129, 257), (257, 129)), ((255, 520),), ((512, 512), (520, 768), (768, 513)),
                                    ((1030, 512), (77, 200), (300, 300)), tuple((96 + 8 * i, 160) for i in range(11))], ids=str)  # fmt: skip
def test_grouped_newton_schulz_step(tile, shapes):
    """Several shapes (up to eleven: more than one launch holds) in one chain, both orientations, ragged tiles.  The iterate is
    read back from a step with polynomial 1 (an identity), then one step with all three coefficients is compared with fp64
    products of the same bf16 operands: what remains is the order of fp32 sums, which may move a value by one bf16 rounding
    (2^-8) in S, in the polynomial and in the result."""
    ext = ops.load()
    ext.set_ns_gemm_tile(tile)
    try:
        gen = torch.Generator(DEV).manual_seed(3)
        mats = [[torch.randn(s, device=DEV, generator=gen) for _ in range(2)] for s in shapes]
        norms = torch.stack([m.square().sum() for pair in mats for m in pair])
        at = [range(2 * k, 2 * k + 2) for k in range(len(shapes))]

        def go(coeffs):
            outs = [torch.full((2, *s), float("nan"), device=DEV) for s in shapes]
            ops.newton_schulz_groups([(m, i, o, 1.0, 7 + k) for k, (m, i, o) in enumerate(zip(mats, at, outs))], norms, coeffs)
            ops.check_status()
            return outs

        start, got = go([(1.0, 0.0, 0.0)]), go([(3.0, -4.0, 2.0)])
    finally:
        ext.set_ns_gemm_tile(0)
    for m, x, y in zip(mats, start, got):
        want_x = torch.stack(m) / torch.stack(m).norm(dim=(-2, -1), keepdim=True)
        assert (x - want_x).abs().max() <= want_x.abs().max() * 2**-7  # stochastic rounding to bf16
        flip = (lambda t: t.mT) if x.shape[-2] > x.shape[-1] else (lambda t: t)
        want = flip(_poly_oracle(flip(x.double()), 3.0, -4.0, 2.0))
        err = (y.double() - want).abs().max() / want.abs().max()
        assert err < 3 * 2**-8, err
        assert (y.double() - want).norm() / want.norm() < 2**-9


def test_stage_ranges_of_a_muon_step():
    """The names that a profiler filter would look for: one range each, whatever the number of shape buckets."""
    from heavyball_b200.utils import tracing

    params = [torch.nn.Parameter(torch.randn(s, device=DEV)) for s in ((64, 128), (96, 64), (128, 128))]
    opt = hb.Muon(params, lr=1e-2)
    for step in range(2):  # the first step creates the state
        for p in params:
            p.grad = torch.randn_like(p)
        if step:
            tracing.enable(True, record=True)
            tracing.seen.clear()
        try:
            opt.step()
        finally:
            tracing.enable(False)
    assert tracing.seen == ["momentum", "newton_schulz", "update"]
    tracing.seen.clear()


# ---------------------------------------------------------------------------------------- triangular leaves


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 95, 127, 128])
def test_cholesky_leaf_at_sub_block_edges(n):
    """Factor and inverse of one leaf at sizes around its 32-wide sub-blocks, for condition numbers up to 1e4: a backward
    stable factorisation reproduces the matrix to n eps and the inverse to n eps times the condition number of the factor."""
    ext = ops.load()
    gen = torch.Generator(DEV).manual_seed(n)
    q = torch.linalg.qr(torch.randn(3, n, n, device=DEV, generator=gen, dtype=torch.float64))[0]
    lam = torch.logspace(0, -4 if n > 1 else 0, n, device=DEV, dtype=torch.float64)
    g = ((q * lam) @ q.mT).float()
    g = (g + g.mT) / 2
    r, info = torch.zeros_like(g), torch.zeros(3, dtype=torch.int32, device=DEV)
    inv = torch.full((3, 1, 128, 128), float("nan"), device=DEV)
    ext.chol_inv_leaf(g, r, inv, 0, n, info)
    assert info.sum().item() == 0
    assert torch.equal(r, r.triu())
    eps = 2.0**-23
    assert (r.double().mT @ r.double() - g.double()).abs().max().item() < 8 * n * eps
    x = inv[:, 0, :n, :n].double()
    assert (x @ r.double() - torch.eye(n, device=DEV, dtype=torch.float64)).abs().max().item() < 8 * n * eps * 1e2
    assert torch.equal(ext.tri_inv_blocks(r)[:, 0, :n, :n], inv[:, 0, :n, :n])
    bad = g.clone()
    bad[1, n // 2, n // 2] = -1.0
    ext.chol_inv_leaf(bad, r, inv, 0, n, info)
    assert info.tolist() == [0, 1, 0]


def _factor(gen, b, n):
    """Statistics whose eigenbasis is known to a few percent, and that basis."""
    q = torch.linalg.qr(torch.randn(b, n, n, device=DEV, generator=gen))[0]
    noise = torch.randn(b, n, n, device=DEV, generator=gen) * 0.02 / n**0.5
    return (q * torch.logspace(1, 0, n, device=DEV)) @ q.mT + noise + noise.mT, q


def _copies(items):
    clone = lambda xs: [None if x is None else x.clone() for x in xs]  # noqa: E731
    return [(clone(g), clone(q), m.clone()) for g, q, m in items]


def _ladder(monkeypatch):
    """An empty ladder memory; returns the list that the calls of the factorisation are added to as (matrices, rounds)."""
    from heavyball_b200.utils import orthogonal

    calls, run = [], orthogonal._cholesky_qr2_replayed
    monkeypatch.setattr(orthogonal, "_cholesky_qr2_replayed", lambda x, rounds=0: calls.append((x.shape[0], rounds)) or run(x, rounds))
    monkeypatch.setattr(orthogonal, "_cholqr_level", {})
    monkeypatch.setattr(orthogonal, "_cholqr_wins", {})
    return calls


@pytest.mark.parametrize("limit", [None, 256 * 256 * 5, 1])
def test_eigenbases_of_several_buckets_refresh_together(limit, monkeypatch):
    """One joint refresh of three buckets (shared sizes, one factor missing) against the bucket-by-bucket definition; ``limit``:
    elements of a joint batch (the default, room for two of the three members of one size, room for none)."""
    from heavyball_b200.utils import soap

    gen = torch.Generator(DEV).manual_seed(5)
    items = []
    for b, (r, c) in ((2, (256, 256)), (3, (256, 384)), (1, (384, None))):
        gl, ql = _factor(gen, b, r)
        gr, qr = _factor(gen, b, c) if c else (None, None)
        items.append(([gl, gr], [ql, qr], torch.randn(b, r, c or 64, device=DEV, generator=gen)))
    want = _copies(items)
    for g, q, m in want:
        utils.get_orthogonal_matrix_QR(g, q, m)
    if limit is not None:
        monkeypatch.setattr(soap, "_JOINT_REFRESH_ELEMENTS", limit)
    calls = _ladder(monkeypatch)
    utils.refresh_eigenbases(items)
    assert sorted(n for n, _ in calls) == {None: [4, 7], 1: [1, 2, 2, 3, 3]}.get(limit, [1, 3, 3, 4])
    for (_, q, m), (_, q0, m0) in zip(items, want):
        for x, y in zip([*q, m], [*q0, m0]):
            if x is not None:
                torch.testing.assert_close(x, y, rtol=0, atol=2e-4)


@pytest.mark.parametrize("n", [128, 256, 384])
def test_a_rank_deficient_factor_does_not_change_how_the_others_refresh(n, monkeypatch):
    """Statistics with rows of zeros (a dead head) in one of three buckets.  The other two take the variants and get the bases that
    they get without it; n = 128 lies below the whole-matrix factorisation and takes the panel-wise one."""
    gen = torch.Generator(DEV).manual_seed(n)
    items = []
    for b in (2, 1, 3):
        g, q = _factor(gen, b, n)
        items.append(([g, None], [q, None], torch.randn(b, n, 64, device=DEV, generator=gen)))
    items[1][0][0][:, n // 2 :] = 0
    items[1][0][0][:, :, n // 2 :] = 0
    want = _copies([items[0], items[2]])
    for g, q, m in want:
        utils.get_orthogonal_matrix_QR(g, q, m)
    calls = _ladder(monkeypatch)
    eye = torch.eye(n, device=DEV)
    for again in range(3):  # eager, captured and replayed; the first refresh finds out, the later ones know
        before, now = len(calls), _copies(items)
        utils.refresh_eigenbases(now)
        assert all(size == 1 for size, rounds in calls[before:] if rounds), calls  # only the deficient bucket climbs
        for (_, q, m), (_, q0, m0) in zip([now[0], now[2]], want):
            torch.testing.assert_close(q[0], q0[0], rtol=0, atol=2e-5)
            torch.testing.assert_close(m, m0, rtol=0, atol=2e-4)
            assert (q[0].mT @ q[0] - eye).abs().max().item() < 1e-4
        assert all(torch.isfinite(q[0]).all() for _, q, _ in now)
