"""The kernels for small calls (mma.sync on 32 x 32 tiles) against float64: at the edges of their tiles, for every layout of the
operands that they fetch, with impossible states, supplied and returned column maxima, and against the tcgen05 kernels."""

import pytest
import torch

from oracle import logspace_oracle as orc
from triturus_b200 import _native

# Plain TF32 rounds both operands of a product to nearest at 10 fraction bits: off by 2^-11 of themselves at most each, and
# exp(b - m) by ulps.  3xTF32: sums of at most 512 (lm2exp) or 128 (lt2exp) terms; the products' low parts are cut at 2^-11 of
# 2^-11, and a sum of 64 MMAs, each truncated, in eight partial sums drifts by 8 * 2^-23.
TOL = {"tf32": 2 * 2.0**-11 + 1e-5, "3xtf32": 1e-5}
# The tcgen05 kernels round one operand and truncate the other, 2^-11 + 2^-10, and the above on this side.
TOL_BOTH = {"tf32": 2.0**-11 + 2.0**-10 + TOL["tf32"], "3xtf32": 1.1e-4}


def _views(t):
    """`t` in the layouts that a caller may pass: contiguous, the last two dimensions swapped in memory, every second element of
    a wider tensor, at an odd base, and with an odd row pitch."""
    wide = torch.zeros(*t.shape[:-1], 2 * t.shape[-1], device=t.device)
    wide[..., ::2] = t
    shifted = torch.zeros(t.numel() + 1, device=t.device)
    shifted[1:] = t.flatten()
    pitched = torch.zeros(*t.shape[:-1], t.shape[-1] + 1 + t.shape[-1] % 2, device=t.device)
    pitched[..., : t.shape[-1]] = t
    return [t, t.transpose(-1, -2).contiguous().transpose(-1, -2), wide[..., ::2], shifted[1:].view(t.shape), pitched[..., : t.shape[-1]]]


def _check(got, want, tol):
    assert torch.equal(got.cpu() == float("-inf"), want == float("-inf")) and not torch.isnan(got).any()
    fin = torch.isfinite(want)
    err = (got.cpu().double() - want).abs()[fin]
    tol = tol + 2.0**-22 * want.abs()[fin]
    assert (err <= tol).all(), (err - tol).max()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["tf32", "3xtf32"])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 33, 9, 31), (3, 32, 8, 64), (2, 31, 7, 33), (1, 64, 64, 96), (5, 40, 130, 44),
                                   (1, 70, 511, 66), (1, 32, 512, 32)], ids=str)  # fmt: skip
def test_lm2exp(shape, precision):
    import triturus_b200 as tb

    R, I, J, K = shape
    for odd in (0, 1):
        assert _native.LIB.triturus_b200_lm2exp_direct(*shape, int(precision == "3xtf32"), 0, odd) == 1
    g = torch.Generator().manual_seed(sum(shape))
    a = torch.rand(R, I, J, generator=g)
    b = torch.randn(R, J, K, generator=g) * 4.0 + 100.0 * torch.randn(R, 1, K, generator=g)
    b[torch.rand(R, J, K, generator=g) < 0.02] = float("-inf")
    b[0, :, K - 1] = float("-inf")
    a[R - 1, I - 1] = 0.0
    want = orc.lm2exp_fp64(a, b)
    first = None
    for av in _views(a.cuda()):
        for bv in _views(b.cuda()):
            got = tb.lm2exp(av, bv, precision=precision)
            first = got if first is None else first
            assert torch.equal(got, first)  # the layout does not matter, bit for bit
    _check(first, want, TOL[precision])
    ad, bd = a.cuda(), b.cuda()
    m = bd.amax(1)
    out, top = tb.lm2exp(ad, bd, precision=precision, b_colmax=m, return_colmax=True)
    assert torch.equal(out, first) and torch.equal(top, out.amax(1))
    if R > 1:
        same = tb.lm2exp(ad[:1].expand(R, I, J), bd[:1].expand(R, J, K), precision=precision)  # stride 0
        assert torch.equal(same, first[:1].expand(R, I, K))
    ref = tb.lm2exp(ad, bd, precision=precision, variant=1281)
    _check(ref, first.cpu().double(), TOL_BOTH[precision])
    tb.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["tf32", "3xtf32"])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 1), (2, 33, 3, 9, 31), (1, 32, 9, 8, 64), (2, 31, 17, 7, 33), (1, 40, 65, 33, 36), (1, 64, 50, 50, 100),
                                   (1, 20, 128, 16, 32), (3, 75, 50, 50, 100)], ids=str)  # fmt: skip
def test_lt2exp(shape, precision):
    import triturus_b200 as tb

    R, S, I, J, K = shape
    for odd in (0, 1):
        assert _native.LIB.triturus_b200_lt2exp_direct(*shape, int(precision == "3xtf32"), 0, odd) == 1
    g = torch.Generator().manual_seed(sum(shape))
    w = torch.rand(R, S, I, J, generator=g)
    a = torch.randn(R, I, K, generator=g) * 4.0 + 100.0 * torch.randn(R, 1, K, generator=g)
    b = torch.randn(R, J, K, generator=g) * 4.0 + 100.0 * torch.randn(R, 1, K, generator=g)
    a[torch.rand(R, I, K, generator=g) < 0.02] = float("-inf")
    b[0, :, K - 1] = float("-inf")
    w[R - 1, S - 1] = 0.0
    want = orc.lt2exp_fp64(w, a, b)
    wd, ad, bd = w.cuda(), a.cuda(), b.cuda()
    first = tb.lt2exp(wd, ad, bd, precision=precision)
    _check(first, want, TOL[precision])
    for av, bv in zip(_views(ad), reversed(_views(bd))):
        assert torch.equal(tb.lt2exp(wd, av, bv, precision=precision), first)
    flat = torch.zeros(w.numel() + 1, device="cuda")
    flat[1:] = wd.flatten()
    assert torch.equal(tb.lt2exp(flat[1:].view(w.shape), ad, bd, precision=precision, mode="unsplit"), first)
    out, top = tb.lt2exp(wd, ad, bd, precision=precision, a_colmax=ad.amax(1), b_colmax=bd.amax(1), return_colmax=True)
    assert torch.equal(out, first) and torch.equal(top, out.amax(1))
    ref = tb.lt2exp(wd, ad, bd, precision=precision, variant=11281)
    _check(ref, first.cpu().double(), TOL_BOTH[precision])
    tb.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["tf32", "3xtf32"])
def test_lt2exp_weights_whose_row_sums_overflow(precision):
    """sum_j w exp(b - mb) of one i is beyond fp32, the result is not: the factor exp(a - ma) belongs to the terms.  Impossible and
    unlikely states, on every i that a warp takes."""
    import triturus_b200 as tb

    R, S, I, J, K = 1, 40, 20, 12, 33
    assert _native.LIB.triturus_b200_lt2exp_direct(R, S, I, J, K, int(precision == "3xtf32"), 0, 0) == 1
    w = torch.full((R, S, I, J), 3e38)
    w[:, :, ::5] = 1.0  # the states of these i are the likely ones
    a = torch.full((R, I, K), float("-inf"))
    a[:, 1::5] = -60.0
    a[:, ::5] = 0.0
    b = torch.zeros(R, J, K)
    want = orc.lt2exp_fp64(w, a, b)
    assert want.isfinite().all()
    _check(tb.lt2exp(w.cuda(), a.cuda(), b.cuda(), precision=precision), want, TOL[precision])
    tb.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["tf32", "3xtf32"])
def test_largest_weights(precision):
    """Weights between the largest tf32 value and the largest float, which rounding to nearest would make infinite."""
    import triturus_b200 as tb

    top = torch.finfo(torch.float32).max
    a = torch.zeros(1, 3, 9)
    a[0, 0, 0], a[0, 1, 5], a[0, 2, 3] = top, top * (1 - 2.0**-13), float("inf")
    b = torch.zeros(1, 9, 33)
    w, x, y = a.view(1, 3, 3, 3), torch.zeros(1, 3, 33), torch.zeros(1, 3, 33)
    for got in (tb.lm2exp(a.cuda(), b.cuda(), precision=precision), tb.lt2exp(w.cuda(), x.cuda(), y.cuda(), precision=precision)):
        _check(got[:, :2], orc.lm2exp_fp64(a, b)[:, :2], TOL[precision])
        assert not got[:, 2].isfinite().any()  # infinity stays what it is (3xTF32: no number, its low part is none)
    tb.check_status()


def test_which_calls_are_small():
    """Explicit variants run what they name, and the rules keep to sizes that the kernels can hold."""
    lm, lt = _native.LIB.triturus_b200_lm2exp_direct, _native.LIB.triturus_b200_lt2exp_direct
    assert lm(4, 256, 256, 256, 0, 0, 0) == 1 and lm(4, 256, 256, 256, 0, 201281, 0) == 0
    assert lm(32, 1024, 1024, 1024, 1, 0, 0) == 0 and lm(1, 1, 513, 1, 0, 0, 0) == 0
    assert lm(24, 150, 101, 203, 1, 0, 1) == 1 and lm(0, 1, 1, 1, 0, 0, 0) < 0
    assert lt(3, 75, 50, 50, 100, 1, 0, 1) == 1 and lt(3, 75, 50, 50, 100, 1, 10000, 1) == 1
    assert lt(3, 75, 50, 50, 100, 1, 99990000, 1) == 0 and lt(3, 75, 50, 50, 100, 1, 11281, 1) == 0
    assert lt(1, 256, 256, 256, 256, 1, 0, 0) == 0 and lt(1, 1, 128, 128, 1, 0, 0, 0) == 0
    # several waves of blocks, one per SM, and contractions of few k-blocks: the tcgen05 kernels are faster
    for shape, precision in (((4, 259, 112, 36, 44), 0), ((34, 2, 37, 60, 108), 1), ((64, 56, 4, 32, 148), 0), ((16, 97, 3, 4, 460), 0)):
        assert lt(*shape, precision, 0, 0) == 0
    assert lt(4, 259, 112, 36, 44, 0, 10000, 0) == 1  # (never split)
    for shape in ((1, 1, 129, 1, 1), (1, 1, 1, 129, 1)):
        assert lt(*shape, 0, 0, 0) == 0


@pytest.mark.gpu
def test_calls_that_the_extension_leaves_to_python():
    """Small calls take the extension module; what it does not recognise behaves as without it: checks, modes, other streams
    and subclasses."""
    import triturus_b200 as tb

    g = torch.Generator().manual_seed(3)
    a, b = torch.rand(2, 40, 24, generator=g).cuda(), torch.randn(2, 24, 50, generator=g).cuda()
    w, x, y = torch.rand(2, 20, 6, 7, generator=g).cuda(), torch.randn(2, 6, 50, generator=g).cuda(), torch.randn(2, 7, 50, generator=g).cuda()
    host = _native.HOST
    out, lt = tb.lm2exp(a, b), tb.lt2exp(w, x, y)
    assert torch.equal(host.lm2exp(a, b, 1, 0), out) and torch.equal(host.lt2exp(w, x, y, 1, 0), lt)
    assert host.lm2exp(a, b, 1, 1281) is None and host.lm2exp(a, b, -1, 0) is None and host.lt2exp(w, x, y, 1, 11281) is None
    assert host.lm2exp(a, b[:, :23], 1, 0) is None and host.lm2exp(a.double(), b.double(), 1, 0) is None
    assert host.lm2exp(a.cpu(), b.cpu(), 1, 0) is None and host.lm2exp(a, None, 1, 0) is None
    assert host.lm2exp(a[:, :0], b, 1, 0) is None
    assert host.lm2exp(torch.rand(64, 512, 256, device="cuda"), torch.rand(64, 256, 512, device="cuda"), 1, 0) is None
    with pytest.raises(AssertionError):
        tb.lm2exp(a, b[:, :23])
    with pytest.raises(ValueError):
        tb.lm2exp(a, b, precision="fp32")
    with pytest.raises(RuntimeError):  # I and J are no single dimension
        tb.lt2exp(torch.rand(2, 20, 7, 6, device="cuda").transpose(2, 3), x, y)
    assert torch.equal(tb.lm2exp(a.requires_grad_(), b), out) and not tb.lm2exp(a, b).requires_grad
    with torch.inference_mode():
        assert torch.equal(tb.lm2exp(a * 1, b * 1), out)
    with torch.device("cuda"):  # a function mode: through Python
        assert host.lm2exp(a, b, 1, 0) is None and torch.equal(tb.lm2exp(a, b), out)

    class Sub(torch.Tensor):
        pass

    assert host.lm2exp(b.as_subclass(Sub), b, 1, 0) is None
    with pytest.raises(Exception):
        torch.vmap(lambda u: tb.lm2exp(u, b))(torch.stack([a, a]))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        again = tb.lm2exp(a, b)
    torch.cuda.synchronize()
    assert torch.equal(again, out)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        held = tb.lm2exp(a, b)
        held_lt = tb.lt2exp(w, x, y)
    held.zero_(), held_lt.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(held, out) and torch.equal(held_lt, lt)
    tb.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_odd_operands_of_larger_calls_are_copied(precision):
    """Above the line of operations where padded copies are faster the extension leaves a call with operands that no tensor map
    describes to Python, which makes them (R6 511^3 in 3xTF32: 43 us with them, 90 without); below it, and for views that
    torch would have to copy, it takes the call."""
    I, J, K = 320, 301, 511
    for R, small in ((4, True), (12, False)):  # 3.9e8 and 1.2e9 operations
        assert _native.LIB.triturus_b200_lm2exp_direct(R, I, J, K, precision, 0, 1) == 1
        a, b = torch.rand(R, I, J, device="cuda"), torch.randn(R, J, K, device="cuda")
        a4, b4 = torch.zeros(R, I, J + 3, device="cuda")[..., :J], torch.zeros(R, J, K + 1, device="cuda")[..., :K]
        a4.copy_(a), b4.copy_(b)
        for x, y in ((a, b), (a, b4), (a4, b)):
            assert (_native.HOST.lm2exp(x, y, precision, 0) is not None) == small
        out = _native._lm2exp_impl(a, b, precision, 0)
        assert torch.allclose(out, torch.log(torch.bmm(a.double(), b.double().exp())).float(), rtol=0, atol=2e-3)
    wide = torch.randn(R, J, 2 * K, device="cuda")[..., ::2]
    assert _native.HOST.lm2exp(a4, wide, precision, 0) is not None


@pytest.mark.gpu
def test_transposed_operands_of_larger_calls_stay_with_the_tensor_maps():
    """Copies of 4 bytes cost the direct kernel more than the kernel that reads transposed views through tensor maps (R16 256^3 in
    3xTF32 21 us, direct 50): fewer such calls are small ones."""
    for R, precision, takes in ((16, 1, (False, False)), (12, 0, (False, False)), (4, 0, (True, True)), (4, 1, (True, True))):
        a, b = torch.rand(R, 256, 256, device="cuda"), torch.randn(R, 256, 256, device="cuda")
        at, bt = a.transpose(1, 2), b.transpose(1, 2)
        got = [_native.HOST.lm2exp(*x, precision, 0) for x in ((a, bt), (at, bt))]
        assert tuple(x is not None for x in got) == takes
        assert got[0] is None or torch.equal(got[0], _native.HOST.lm2exp(a, bt.contiguous(), precision, 0))


@pytest.mark.gpu
def test_threads_run_while_a_launch_waits_for_the_queue():
    """More calls than the queue of a stream holds, behind a kernel of about a second: while a call waits in its launch another
    Python thread goes on."""
    import threading
    import time

    import triturus_b200 as tb

    a, b = torch.rand(2, 40, 24, device="cuda"), torch.randn(2, 24, 50, device="cuda")
    w, x, y = torch.rand(2, 20, 6, 7, device="cuda"), torch.randn(2, 6, 50, device="cuda"), torch.randn(2, 7, 50, device="cuda")
    for call in (lambda: _native.HOST.lm2exp(a, b, 1, 0), lambda: _native.HOST.lt2exp(w, x, y, 1, 0)):
        assert call() is not None
        torch.cuda.synchronize()
        gaps, stop = [0.0], threading.Event()

        def ticks():
            last = time.perf_counter()
            while not stop.is_set():
                time.sleep(1e-3)
                now = time.perf_counter()
                gaps.append(now - last)
                last = now

        other = threading.Thread(target=ticks)
        other.start()
        torch.cuda._sleep(int(1.5e9))  # 0.75 s at 2 GHz, at most twice that
        start = time.perf_counter()
        for _ in range(3000):
            call()
        waited = time.perf_counter() - start
        stop.set()
        other.join()
        torch.cuda.synchronize()
        assert waited > 0.4, waited  # (the launches did wait, or the test says nothing)
        assert max(gaps) < 0.5 * waited, (max(gaps), waited)
    tb.check_status()
