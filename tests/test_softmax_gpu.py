"""softmax / logsoftmax kernels against the CPU oracle (the comparison the reference's
test/ext_cuda/softmax.jl makes between its CPU and CUDA methods)."""
import numpy as np
import pytest
import torch

import nnlib_jl_b200 as nb
from nnlib_jl_b200 import softmax as SM
from oracle import softmax_oracle as S

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
TOL = {torch.float32: 2e-6, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


def _dev(a, dtype):
    return nb.jl_from_numpy(np.asarray(a, dtype=np.float32), device=DEV).to(dtype) if dtype != torch.float32 \
        else nb.jl_from_numpy(np.asarray(a, dtype=np.float32), device=DEV)


def _round(a, dtype):
    return torch.from_numpy(np.asarray(a, dtype=np.float32)).to(dtype).float().numpy()


def _as_cm(t, dtype):
    """column-major device tensor of element type dtype"""
    out = nb.jl_empty(tuple(t.shape), dtype, DEV)
    out.copy_(t)
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape,dims", [
    ((5, 7), 1), ((5, 7), 2), ((300, 33), 1), ((2000, 9), 1), ((4100, 3), 1),      # warp- and block-per-column
    ((256, 10, 32), 2), ((16, 5, 3, 4), 3), ((16, 5, 3, 4), 4), ((7, 9), None), ((3, 4), 3), ((6, 5, 4), (1, 2)), ((6, 5, 4), (2, 3)),
])
def test_forward_and_pullbacks_match_the_oracle(dtype, shape, dims):
    rng = np.random.default_rng(5)
    xn = _round(3.0 * rng.standard_normal(shape), dtype)
    dyn = _round(rng.standard_normal(shape), dtype)
    x, dy = _as_cm(_dev(xn, dtype), dtype), _as_cm(_dev(dyn, dtype), dtype)
    tol = TOL[dtype]
    y = SM.softmax(x, dims=dims)
    ly = SM.logsoftmax(x, dims=dims)
    yo, lyo = S.softmax(xn, dims), S.logsoftmax(xn, dims)
    np.testing.assert_allclose(nb.jl_to_numpy(y), yo, atol=tol, rtol=tol)
    np.testing.assert_allclose(nb.jl_to_numpy(ly), lyo, atol=tol * max(1.0, np.abs(lyo).max()), rtol=tol)
    # pullbacks take the device's own (rounded) y, like the reference's rrule does
    yr, lyr = nb.jl_to_numpy(y), nb.jl_to_numpy(ly)
    dx = SM.softmax_pullback(dy, y, dims=dims)
    np.testing.assert_allclose(nb.jl_to_numpy(dx), S.softmax_pullback(dyn, yr, dims), atol=4 * tol, rtol=4 * tol)
    dlx = SM.logsoftmax_pullback(dy, ly, dims=dims)
    want = S.logsoftmax_pullback(dyn, lyr, dims)
    np.testing.assert_allclose(nb.jl_to_numpy(dlx), want, atol=4 * tol * max(1.0, np.abs(want).max()), rtol=4 * tol)


@pytest.mark.parametrize("dtype,n,cols", [
    (torch.bfloat16, 16392, 593),     # one packet more than 256 threads hold
    (torch.float16, 32768, 592),      # all eight packets of 512 threads
    (torch.float32, 16388, 601),      # one packet beyond that: 1024 threads, two columns arriving
    (torch.bfloat16, 57344, 593),     # all seven of those
    (torch.bfloat16, 57352, 593),     # longer than that, the other kernel
    (torch.bfloat16, 16392, 591),     # too few columns
])
def test_long_columns_arriving_ahead(dtype, n, cols):
    """Long contiguous columns, among them ones with +Inf, -Inf and NaN entries, against the same columns in a batch too
    small for them to be fetched ahead (torch's Float64 softmax for the ordinary ones)."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    t = torch.empty((cols, n), device=DEV).normal_(0, 3, generator=gen)
    inf = float("inf")
    t[5, 17], t[5, n - 1], t[300, 3], t[590, :], t[7, 0] = inf, inf, float("nan"), -inf, -inf
    x = t.to(dtype).t()
    few = [0, 5, 7, 148, 300, 295, 296, cols - 1, 590]
    for f, ref in ((SM.softmax, torch.softmax), (SM.logsoftmax, torch.log_softmax)):
        y = f(x)
        sub = _as_cm(x[:, few], dtype)
        assert torch.allclose(y[:, few].float(), f(sub).float(), rtol=2 * TOL[dtype], atol=1e-6 if f is SM.softmax else 2 * TOL[dtype],
                              equal_nan=True)
        want = ref(x[:, [0, 7, 148, 296]].double(), 0)
        got = y[:, [0, 7, 148, 296]].double()
        assert torch.allclose(got, want, rtol=TOL[dtype] if dtype != torch.float32 else 1e-5, atol=1e-9 if dtype != torch.float16 else 6e-8)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,cols", [(32776, 592), (50000, 700), (57344, 592), (57352, 592), (50000, 300)])
def test_softmax_of_very_long_16_bit_columns_is_rounded_once(dtype, n, cols):
    """Columns that no kernel keeps the exponentials of, fetched ahead or not: half a unit of the element type, and 2^-16
    for the exponentials and their Float32 sum."""
    gen = torch.Generator(device="cuda").manual_seed(n + cols)
    x = torch.empty((cols, n), device=DEV).normal_(0, 3, generator=gen).to(dtype).t()
    y = SM.softmax(x).t().double()
    want = torch.softmax(x.t().double(), 1)
    digits, sub = (8, 0.0) if dtype == torch.bfloat16 else (11, 2.0 ** -25)
    half = torch.clamp(torch.ldexp(torch.ones_like(want), torch.frexp(want).exponent - 1 - digits), min=sub)
    assert bool(((y - want).abs() <= half + 2.0 ** -16 * want).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape,dims", [((300, 33), 1), ((70000, 3), 1), ((64, 50, 4), 2)])
def test_in_place_forms(dtype, shape, dims):
    """softmax!(x, x) and the pullbacks written over dy or y (src/softmax.jl:66, 98-101): the same values as
    the out-of-place calls, for a warp per column, a block per column with re-read columns, and the
    strided kernel."""
    rng = np.random.default_rng(7)
    x = _as_cm(_dev(_round(3.0 * rng.standard_normal(shape), dtype), dtype), dtype)
    dy = _as_cm(_dev(_round(rng.standard_normal(shape), dtype), dtype), dtype)
    for fwd, bwd in ((SM.softmax, SM.softmax_pullback), (SM.logsoftmax, SM.logsoftmax_pullback)):
        y = fwd(x, dims=dims)
        xc = x.clone()
        assert fwd(xc, dims=dims, out=xc) is xc
        assert torch.equal(xc, y)
        dx = bwd(dy, y, dims=dims)
        dyc, yc = dy.clone(), y.clone()
        bwd(dyc, y, dims=dims, out=dyc)
        bwd(dy, yc, dims=dims, out=yc)
        assert torch.equal(dyc, dx) and torch.equal(yc, dx)


def test_inf_nan_table_on_device():
    # test/softmax.jl:62-75 and the masked-input regression of test/ext_cuda/softmax.jl:34-78
    f, inf, nan = np.float32, np.inf, np.nan
    for xn in (f([[1, 2], [3, inf]]), f([[1, -inf], [3, inf]]), f([[1, inf], [3, inf]]), f([[1, 2], [3, nan]]),
               f([[-inf, 1], [-inf, 2]]), f([[-1000, 1], [-1000, -inf]])):
        for dims in (1, 2):
            x = _as_cm(_dev(xn, torch.float32), torch.float32)
            np.testing.assert_allclose(nb.jl_to_numpy(SM.softmax(x, dims=dims)), S.softmax(xn, dims), rtol=1e-6, atol=1e-7)
            got, want = nb.jl_to_numpy(SM.logsoftmax(x, dims=dims)), S.logsoftmax(xn, dims)
            np.testing.assert_allclose(got, want, rtol=1e-6, atol=1e-6)
    # masked entries are exactly zero, the others sum to one
    rng = np.random.default_rng(6)
    xn = rng.standard_normal((64, 50)).astype(np.float32)
    keep = rng.random((64, 50)) > 0.4
    keep[0] = True
    xm = np.where(keep, xn, -np.inf).astype(np.float32)
    y = nb.jl_to_numpy(SM.softmax(_as_cm(_dev(xm, torch.float32), torch.float32)))
    assert ((y > 0) == keep).all()
    np.testing.assert_allclose(y.sum(0), 1.0, rtol=1e-5)


def test_argument_checks():
    x = nb.jl_zeros((4, 5), torch.float32, DEV)
    with pytest.raises(nb.ArgumentError):
        SM.softmax(x, dims=0)
    with pytest.raises(nb.ArgumentError):
        SM.softmax(nb.jl_zeros((4, 5, 6), torch.float32, DEV), dims=(1, 3))
    with pytest.raises(nb.ArgumentError):
        SM.softmax_pullback(nb.jl_zeros((4, 6), torch.float32, DEV), x)
    with pytest.raises(TypeError):
        SM.softmax(torch.zeros(3, 3))
    assert tuple(SM.softmax(nb.jl_zeros((0, 5), torch.float32, DEV)).shape) == (0, 5)


@pytest.mark.parametrize("seed", range(40))
def test_random_shapes_and_dims_match_the_oracle(seed):
    """Seeded random draws: element type, rank 1 to 4, sizes that land on every kernel variant (a warp, a block
    or a large block per column, cached or re-read columns, the strided kernel), any run of consecutive dims,
    forward / log forward and both pullbacks, out of place and in place."""
    rng = np.random.default_rng(12000 + seed)
    dtype = [torch.float32, torch.float16, torch.bfloat16][seed % 3]
    rank = int(rng.integers(1, 5))
    first = int(rng.choice([1, 3, 8, 33, 64, 257, 512, 1000, 2048, 4100, 9000, 20000]))
    rest = [int(rng.integers(1, 7)) for _ in range(rank - 1)]
    shape = tuple([min(first, max(1, 600000 // int(np.prod(rest)))) if rest else first] + rest)
    lo = int(rng.integers(1, rank + 1)); hi = int(rng.integers(lo, rank + 1))
    dims = lo if lo == hi else tuple(range(lo, hi + 1))
    xn = _round(3.0 * rng.standard_normal(shape), dtype)
    dyn = _round(rng.standard_normal(shape), dtype)
    x, dy = _as_cm(_dev(xn, dtype), dtype), _as_cm(_dev(dyn, dtype), dtype)
    tol = TOL[dtype]
    what = f"seed {seed}: {dtype} shape {shape} dims {dims}"
    y, ly = SM.softmax(x, dims=dims), SM.logsoftmax(x, dims=dims)
    yo, lyo = S.softmax(xn, dims), S.logsoftmax(xn, dims)
    np.testing.assert_allclose(nb.jl_to_numpy(y), yo, atol=tol, rtol=tol, err_msg=what)
    np.testing.assert_allclose(nb.jl_to_numpy(ly), lyo, atol=tol * max(1.0, np.abs(lyo).max()), rtol=tol, err_msg=what)
    yr, lyr = nb.jl_to_numpy(y), nb.jl_to_numpy(ly)
    dx = SM.softmax_pullback(dy, y, dims=dims)
    np.testing.assert_allclose(nb.jl_to_numpy(dx), S.softmax_pullback(dyn, yr, dims), atol=4 * tol, rtol=4 * tol, err_msg=what)
    dlx = SM.logsoftmax_pullback(dy, ly, dims=dims)
    want = S.logsoftmax_pullback(dyn, lyr, dims)
    np.testing.assert_allclose(nb.jl_to_numpy(dlx), want, atol=4 * tol * max(1.0, np.abs(want).max()), rtol=4 * tol, err_msg=what)
    # in place: the same values as out of place, bit for bit
    x2 = _as_cm(_dev(xn, dtype), dtype)
    SM.softmax(x2, dims=dims, out=x2)
    assert torch.equal(x2, y), what
    dy2 = _as_cm(_dev(dyn, dtype), dtype)
    SM.softmax_pullback(dy2, y, dims=dims, out=dy2)
    assert torch.equal(dy2, dx), what


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("inner,n,outer", [
    (2, 1, 1),            # smallest
    (7, 65, 3),           # fewer columns than a sector
    (33, 300, 2),         # one column past a block of 32; eight loads in flight and a remainder
    (40, 1500, 1),        # long reduction: 1024 threads
    (70, 63, 400),        # enough columns for four threads each
    (2, 4, 700),          # a column a thread: blocks run across the slices
    (3, 23, 10001),       # 8 + 8 + 4 + 2 + 1 elements, the last block not whole
    (5, 33, 23000),       # ... of more than 100000 columns
    (9, 19, 300),         # four threads a column, across slices
    (33, 130, 600),       # eight threads a column, across slices
    (11, 515, 900),       # the columns of a sector, across slices
    (3, 1025, 90),        # 1024 threads, a slice narrower than a sector
])
@pytest.mark.parametrize("log", [False, True])
def test_strided_reduction_blocks(dtype, inner, n, outer, log):
    rng = np.random.default_rng(inner + n)
    xn = 3 * rng.standard_normal((inner, n, outer)).astype(np.float32)
    dn = rng.standard_normal((inner, n, outer)).astype(np.float32)
    if n > 10:
        xn[0, 3, 0] = np.inf                   # equal shares on the +Inf entries
        xn[1, :, 0] = -np.inf                  # nothing but -Inf: NaN
        xn[-1, 5, -1] = np.nan
    x, dy = (nb.jl_from_numpy(a, dtype=dtype, device="cuda:0") for a in (xn, dn))
    x64, d64 = (t.to(torch.float64) for t in (x, dy))
    fwd, back = (nb.softmax.logsoftmax, nb.softmax.logsoftmax_pullback) if log else (nb.softmax.softmax, nb.softmax.softmax_pullback)
    y = fwd(x, dims=2)
    ok = torch.isfinite(x64).all(dim=1, keepdim=True).expand_as(x64)
    want = torch.log_softmax(x64, 1) if log else torch.softmax(x64, 1)
    # the fast exponential and logarithm: a few 2^-22 of |x| <= 16; one rounding to the element type
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 5e-6
    scale = want.abs().clamp_min(1.0 if log else 0.0)
    assert ((y.double() - want).abs() <= rel * scale + 1e-12)[ok].all()
    if n > 10:
        assert y[0, 3, 0].item() == (0.0 if log else 1.0) and torch.isnan(y[1, :, 0]).all() and torch.isnan(y[-1, :, -1]).all()
    dx = back(dy, y, dims=2)
    y64 = y.double()
    s = (d64 if log else d64 * y64).sum(1, keepdim=True)
    wantd = d64 - torch.exp(y64) * s if log else y64 * (d64 - s)
    size = d64.abs() + (torch.exp(y64) if log else y64) * (d64 if log else d64 * y64).abs().sum(1, keepdim=True) + y64.abs() * d64.abs()
    assert ((dx.double() - wantd).abs() <= 2 * rel * size + 1e-12)[ok].all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("inner,n,outer", [(2, 2, 1000000), (2, 4, 1000000), (5, 5, 300000), (8, 10, 500000)])
def test_short_reductions_of_many_columns_run_at_the_speed_of_memory(dtype, inner, n, outer):
    """A handful of elements per column, few columns per slice: within 12 times of a copy of the array, forward and
    back (two to five times is usual; one block per slice took 50 to 140)."""
    x = torch.randn(outer, n, inner, device="cuda:0").to(dtype).permute(2, 1, 0)
    y = nb.softmax.softmax(x, dims=2)
    other = torch.empty(outer, n, inner, device="cuda:0", dtype=dtype)

    def once(f):
        best = float("inf")
        for _ in range(5):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(4):
                f()
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1) / 4)
        return best

    copy = once(lambda: other.copy_(x.permute(2, 1, 0))) + 0.02     # and 20 us for a call from Python
    assert once(lambda: nb.softmax.softmax(x, dims=2)) < 12 * copy
    assert once(lambda: nb.softmax.softmax_pullback(x, y, dims=2)) < 12 * copy
