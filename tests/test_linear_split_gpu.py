"""Products of a prompt in fp32 on the tensor cores against the sums in 64 bits: no further off than a sum in fp32 may be."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from based_b200 import ops as _ops
    return _ops


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


# edges of the tiles (256 rows; 128 or 256 columns), of a chunk of K (64) and of a run of chunks (128), several weights, more than one
# round of wide tiles, values of several magnitudes
@pytest.mark.parametrize("M,parts,K,scale", [(1, (4,), 8, 1.0), (255, (124,), 64, 1e20), (257, (132,), 72, 1e-20), (300, (16, 240, 8), 136, 1.0),
                                             (999, (256, 256, 512, 4), 192, 1.0), (2048, (1536,), 1024, 1.0), (5000, (1100, 1000), 264, 1.0)])
def test_split_products(ops, M, parts, K, scale):
    from based_b200 import _capi
    g = torch.Generator("cuda").manual_seed(M + K)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, ws, b = r(M, K) * scale, [r(n, K) * 10.0 ** i for i, n in enumerate(parts)], r(sum(parts)) * scale
    got = ops.linear_split(x, ws).split(list(parts), -1)
    for y, w in zip(got, ws):
        ref = x.double() @ w.double().T
        # what is left out of a product 2^-24 of it at most, two sums of at most 128 / 16 steps a run, one rounding a run: measured 1.25e-7 to 1.4e-7
        assert _rel(y, ref) < 4e-7, (_rel(y, ref), _rel(torch.nn.functional.linear(x, w), ref))
    y = ops.linear_split(x, ws, b)
    assert _rel(y, x.double() @ torch.cat(ws).double().T + b.double()) < 4e-7
    assert _capi.read_status() == 0


# What a split may lose shows where nothing cancels: operands of one sign, constant ones, the largest part of a bf16 value (2^-7 - 2^-23 cut
# after it leaves 2^-7), rows of very small and very large values.  Both tiles.
@pytest.mark.parametrize("M,N", [(256, 128), (2048, 1536)])
@pytest.mark.parametrize("K", [8, 200, 1024])
@pytest.mark.parametrize("kind", ["1 + 2^-7 - 2^-23", "0.1", "1 - 2^-24", "positive", "signs", "tiny", "subnormal", "huge", "rows"])
def test_split_products_element_by_element(ops, M, N, K, kind):
    g = torch.Generator("cuda").manual_seed(K)
    x, w = torch.rand(M, K, generator=g, device="cuda") + 0.5, torch.rand(N, K, generator=g, device="cuda") + 0.5
    const = {"1 + 2^-7 - 2^-23": 1 + 2 ** -7 - 2 ** -23, "0.1": 0.1, "1 - 2^-24": 1 - 2 ** -24}.get(kind)
    if const is not None:
        x.fill_(const), w.fill_(const)
    elif kind == "signs":
        x, w = x * torch.randn_like(x).sign(), w * torch.randn_like(w).sign()
    elif kind == "tiny":
        x, w = x * 2.0 ** -118, w * 2.0 ** 30
    elif kind == "subnormal":          # 2^-132 to 2^-131: 18 bits of the operand, exactly
        x, w = x * 2.0 ** -131, w * 2.0 ** 60
    elif kind == "huge":               # the products come near the largest float, their sums do not pass it
        x, w = x * 2.0 ** 100, w * (2.0 ** 26 / K)
    elif kind == "rows":
        x = x * 2.0 ** torch.arange(M, device="cuda").remainder(120).sub(60)[:, None]
        w = w * 2.0 ** torch.arange(N, device="cuda").remainder(100).sub(50)[:, None]
    y, xd, wd = ops.linear_split(x, (w,)), x.double(), w.double()
    ref, room = xd @ wd.T, xd.abs() @ wd.abs().T
    off = ((y.double() - ref).abs() / room).max().item()
    # a product to 2^-24, and 2^-24 more for each of the sums of the runs of 128 values and for what the tensor cores cut in a run
    assert off < 2 ** -24 * (2 + K / 128 + 4), off * 2 ** 24


def test_split_products_of_mixed_magnitudes(ops):
    """Values far below their row's largest: to 2^-133 of it, which bounds what they may add.  A few products carry each sum, so that all of
    the sixteen steps of the tensor cores may cut it, by 2^-23 each."""
    K = 256
    g = torch.Generator("cuda").manual_seed(1)
    x, w = torch.rand(512, K, generator=g, device="cuda") + 0.5, torch.rand(256, K, generator=g, device="cuda") + 0.5
    x[:, 1:] *= 2.0 ** -torch.randint(1, 140, (512, K - 1), generator=g, device="cuda").float()
    w[:, 0], w[:, 1] = 0, 2.0 ** 40      # the row's largest of x meets nothing
    y, ref, room = ops.linear_split(x, (w,)).double(), x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert bool(((y - ref).abs() <= room * 2 ** -23 * (K // 16) + K * 2.0 ** -132 * 2.0 ** 41).all())


def test_split_products_of_special_values(ops):
    """Infinite and undefined sums as torch has them, for both tiles; the largest values do not overflow on the way."""
    for M, N in ((256, 128), (2048, 1536)):
        x, w = torch.randn(M, 200, device="cuda"), torch.randn(N, 200, device="cuda")
        x[3, 5], x[7, 1], x[9, 2], x[13, 199] = float("inf"), float("nan"), 3.4e38, -float("inf")
        w[4] = 0
        w[4, 2], w[6, 7], w[8, 0] = 0.5, 0.0, float("inf")
        y, ref = ops.linear_split(x, (w,)), torch.nn.functional.linear(x, w)
        finite = torch.isfinite(ref)
        assert torch.equal(torch.isnan(y), torch.isnan(ref)) and torch.equal(torch.isfinite(y), finite)
        assert torch.equal(y[torch.isinf(ref)], ref[torch.isinf(ref)])
        assert torch.allclose(y[finite], ref[finite], rtol=1e-4, atol=1e-4)


def test_prompt_routes(ops, monkeypatch):
    """The mixer's projections are two calls of it; a watched projection is still called as a module, and so is one under autocast."""
    from based_b200.mixers import LinearAttention
    m = LinearAttention(512, num_heads=8, layer_idx=0, device="cuda").eval()
    x = torch.randn(2, 1024, 512, device="cuda")
    calls, own = [], ops.linear_split
    monkeypatch.setattr(ops, "linear_split", lambda *a, **k: calls.append(1) or own(*a, **k))
    with torch.inference_mode():
        y = m(x)
        assert len(calls) == 2
        seen = []
        h = m.proj_k.register_forward_hook(lambda *a: seen.append(1))
        z = m(x)
        h.remove()
        assert len(calls) == 3 and len(seen) == 1 and torch.allclose(y, z, rtol=1e-3, atol=1e-4)
        m(x[:, :100])
        assert len(calls) == 3       # few rows: the library
    with pytest.raises(RuntimeError):
        m(x)                         # the kernels have no backward
    assert len(calls) == 3


@pytest.mark.parametrize("M,parts,K", [(24000, (8, 500), 1024), (65536, (64, 64, 132), 512), (30001, (260,), 2048)])
def test_many_rows_share_a_bounded_scratch(ops, M, parts, K):
    """Rows in parts (two to six): the results of smaller calls, and no more memory than the bound."""
    from based_b200 import _capi
    assert 60 << 20 < _capi.lib().based_linear_f32_scratch_bytes(M, sum(parts), K) <= 128 << 20
    g = torch.Generator("cuda").manual_seed(M)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, ws, b = r(M, K), [r(n, K) for n in parts], r(sum(parts))
    with torch.inference_mode():
        torch.cuda.synchronize()
        held = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        y = ops.linear_split(x, ws, b)
        assert torch.cuda.max_memory_allocated() - held <= (128 << 20) + y.numel() * 4 + 4096
        for a in (0, 4096, M // 2 - 300, M - 700):
            ref = x[a:a + 700].double() @ torch.cat(ws).double().T + b.double()
            assert _rel(y[a:a + 700], ref) < 4e-7
        w = torch.cat(ws)
        wide = torch.nn.functional.linear(x, w, b)
        assert float((y - wide).abs().max()) < 1e-4 * float(wide.abs().max())     # every row is there
    assert _capi.read_status() == 0


def test_large_weights_stay_with_the_library(ops):
    x, w = torch.zeros(128, 1024, device="cuda"), torch.zeros(8200, 1024, device="cuda")
    with torch.inference_mode():
        assert ops._split_rows(x, (w[:8192],)) and not ops._split_rows(x, (w,))


def test_projections_with_a_bias(ops):
    """A projection that was replaced by one with a bias keeps it."""
    from based_b200.mixers import LinearAttention
    m = LinearAttention(512, num_heads=8, layer_idx=0, device="cuda").eval()
    x = torch.randn(2, 1024, 512, device="cuda")
    for name in ("proj_q", "proj_k", "proj_v"):
        plain = getattr(m, name)
        biased = torch.nn.Linear(512, plain.out_features, device="cuda")
        with torch.inference_mode():
            biased.weight.copy_(plain.weight)
            biased.bias.fill_(0.5)
            setattr(m, name, biased)
            y = m(x)
            h = biased.register_forward_hook(lambda *a: None)   # watched: called as a module
            assert torch.allclose(y, m(x), rtol=1e-3, atol=1e-4)
            h.remove()
            setattr(m, name, plain)
            assert not torch.allclose(y, m(x), rtol=1e-2, atol=1e-3)


def _set(where, name, value):
    return lambda: setattr(where, name, value)


@pytest.mark.parametrize("allow,forbid", [
    (_set(torch.backends, "fp32_precision", "tf32"), _set(torch.backends, "fp32_precision", "none")),
    (_set(torch.backends.cuda.matmul, "fp32_precision", "tf32"), _set(torch.backends.cuda.matmul, "fp32_precision", "none")),
    (_set(torch.backends.cuda.matmul, "allow_tf32", True), _set(torch.backends.cuda.matmul, "allow_tf32", False)),
    (lambda: torch.set_float32_matmul_precision("high"), lambda: torch.set_float32_matmul_precision("highest"))])
def test_callers_that_let_products_round(ops, monkeypatch, allow, forbid):
    """Who allows TF32 gets the library's one pass over rounded operands, by whichever switch; switched back, the exact products."""
    calls, own = [], ops.linear_split
    monkeypatch.setattr(ops, "linear_split", lambda *a, **k: calls.append(1) or own(*a, **k))
    x, w = torch.randn(1024, 1024, device="cuda"), torch.randn(1024, 1024, device="cuda")
    with torch.inference_mode():
        y = ops.linear(x, w)
        try:
            allow()
            z = ops.linear(x, w)
            assert len(calls) == 1 and torch.equal(z, torch.nn.functional.linear(x, w)) and not torch.equal(y, z)
        finally:
            forbid()
        assert torch.equal(ops.linear(x, w), y) and len(calls) == 2
