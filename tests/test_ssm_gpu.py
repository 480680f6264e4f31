"""Parity of the fused SSM stage (discretise + scan + read out) with the CPU oracle, through the C ABI."""
import numpy as np
import pytest

import oracle as O
from parity import REL_TOL, chan_err, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import pssa_b200
    d = pssa_b200.B200Dispatch(0)
    yield d
    d.close()


def inputs(T, d, s, seed):
    rng = np.random.default_rng(seed)
    delta = np.log1p(np.exp(rng.normal(-2.0, 1.0, (T, d)))).astype(np.float32)  # softplus of a projection
    bp = rng.normal(0, 1, (T, s)).astype(np.float32)
    cp = rng.normal(0, 1, (T, s)).astype(np.float32)
    x = rng.normal(0, 1, (T, d)).astype(np.float32)
    # decay exp(delta*A) mostly in (0.9, 0.999) like the model's log-spaced rates (src/pssa.rs:649-665)
    rates = -np.exp(rng.uniform(np.log(0.005), np.log(0.7), d * s)).astype(np.float32)
    h0 = rng.normal(0, 1, d * s).astype(np.float32)
    return delta, bp, cp, x, rates, h0


SHAPES = [(1, 4, 2), (2, 7, 3), (3, 16, 16), (31, 12, 4), (32, 64, 64), (33, 20, 8), (257, 32, 64), (130, 9, 5),
          (64, 8, 128), (40, 192, 64)]


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("T,d,s", SHAPES)
def test_single_lane_matches_ordered_recurrence(gpu, T, d, s, exact):
    delta, bp, cp, x, rates, h0 = inputs(T, d, s, T * 1000 + d * 10 + s)
    ref_states, ref_y, ref_a, ref_b = O.ssm_forward(delta, bp, cp, x, rates, h0, mode=0)
    y = np.empty((T, d), np.float32)
    states = np.empty((T + 1, d * s), np.float32)
    bar_a = np.empty((T, d * s), np.float32)
    bar_b = np.empty((T, d * s), np.float32)
    gpu.ssm_forward(delta, bp, x, rates, cp, h0, T, d, s, bar_a, bar_b, states, y, exact=exact)
    assert np.array_equal(states[0], h0)
    assert np.array_equal(bar_b.view(np.uint32), ref_b.view(np.uint32))  # one rounded product in both modes
    assert rel_err(bar_a, ref_a) <= (2e-7 if exact else 6e-7)
    tol = 5e-6 if exact else REL_TOL  # CUDA expf (<= 2 ulp) vs glibc expf, both within their documented error
    assert chan_err(states, ref_states, 0) <= tol
    assert chan_err(y, ref_y, 0) <= tol
    # without the tape outputs (the inference form) y is the same
    y2 = np.empty_like(y)
    gpu.ssm_forward(delta, bp, x, rates, cp, h0, T, d, s, None, None, None, y2, exact=exact)
    assert np.array_equal(y2, y)


def test_packed_ragged_lanes_with_an_idle_lane(gpu):
    # lanes as in src/sequence_batch.rs:233-384: packed rows, per-lane carry; an omitted lane keeps its carry
    import torch
    d, s = 48, 16
    lengths = np.array([5, 0, 33, 1, 70], np.uint32)
    offsets = np.concatenate([[0], np.cumsum(lengths)[:-1]]).astype(np.uint32)
    rows = int(lengths.sum())
    delta, bp, cp, x, rates, _ = inputs(rows, d, s, 77)
    carry = np.random.default_rng(1).normal(size=(len(lengths), d * s)).astype(np.float32)
    ref_carry = carry.copy()
    ref_y = O.ssm_lanes(delta, bp, cp, x, rates, ref_carry, offsets, lengths)
    t = {k: torch.from_numpy(v).cuda() for k, v in dict(delta=delta, bp=bp, cp=cp, x=x, rates=rates, carry=carry).items()}
    y = torch.zeros(rows, d, device="cuda")
    gpu.set_stream(torch.cuda.current_stream())
    for exact in (False, True):
        c = t["carry"].clone()
        gpu.ssm_forward_dev(t["delta"], t["bp"], t["cp"], t["x"], t["rates"], c, y, offsets, lengths, rows, d, s,
                            exact=exact)
        torch.cuda.synchronize()
        got_c = c.cpu().numpy()
        assert np.array_equal(got_c[1], carry[1])  # idle lane untouched
        assert chan_err(y.cpu().numpy(), ref_y, 0) <= REL_TOL
        scale = np.maximum(1e-6, np.abs(ref_carry).max())
        assert float(np.max(np.abs(got_c - ref_carry))) / scale <= REL_TOL
    gpu.set_stream(None)


def test_decode_step_shape_one_token_per_lane_with_an_idle_lane(gpu):
    """Every lane one token long (the decode step, which has its own kernel in the fast mode): y and the carries
    match the oracle, the idle lane keeps its carry, and a second step continues from the first."""
    import torch
    for d, s in ((48, 16), (768, 64), (20, 8), (32, 128)):
        lengths = np.array([1, 1, 0, 1, 1, 1], np.uint32)
        offsets = np.concatenate([[0], np.cumsum(lengths)[:-1]]).astype(np.uint32)
        rows = int(lengths.sum())
        carry = np.random.default_rng(d).normal(size=(len(lengths), d * s)).astype(np.float32)
        ref_carry = carry.copy()
        c = torch.from_numpy(carry).cuda()
        gpu.set_stream(torch.cuda.current_stream())
        for step in range(2):
            delta, bp, cp, x, rates, _ = inputs(rows, d, s, 100 + step)
            ref_y = O.ssm_lanes(delta, bp, cp, x, rates, ref_carry, offsets, lengths)
            t = {k: torch.from_numpy(v).cuda() for k, v in dict(delta=delta, bp=bp, cp=cp, x=x, rates=rates).items()}
            y = torch.zeros(rows, d, device="cuda")
            gpu.ssm_forward_dev(t["delta"], t["bp"], t["cp"], t["x"], t["rates"], c, y, offsets, lengths, rows, d, s)
            torch.cuda.synchronize()
            got_c = c.cpu().numpy()
            assert np.array_equal(got_c[2], carry[2])  # idle lane untouched
            assert chan_err(y.cpu().numpy(), ref_y, 0) <= REL_TOL
            scale = np.maximum(1e-6, np.abs(ref_carry).max())
            assert float(np.max(np.abs(got_c - ref_carry))) / scale <= REL_TOL
        gpu.set_stream(None)


def test_continuation_equals_one_pass_bitwise_at_model_size(gpu):
    """Size-independent property at the stacked model's shape (d 768, state 64): running a sequence in two
    calls with the carry handed over gives bit-identical y and carry to one call (src/pssa.rs:1245-1247)."""
    import torch
    lanes, T, d, s = 4, 512, 768, 64
    g = torch.Generator(device="cuda").manual_seed(5)
    delta = torch.nn.functional.softplus(torch.randn(lanes * T, d, device="cuda", generator=g) - 2.0)
    x = torch.randn(lanes * T, d, device="cuda", generator=g)
    bp = torch.randn(lanes * T, s, device="cuda", generator=g)
    cp = torch.randn(lanes * T, s, device="cuda", generator=g)
    rates = -torch.exp(torch.empty(d, s, device="cuda").uniform_(-5.0, -0.4, generator=g))
    off = (np.arange(lanes) * T).astype(np.uint32)
    full = np.full(lanes, T, np.uint32)
    half = np.full(lanes, T // 2, np.uint32)
    gpu.set_stream(torch.cuda.current_stream())
    c1 = torch.zeros(lanes, d * s, device="cuda")
    y1 = torch.zeros(lanes * T, d, device="cuda")
    gpu.ssm_forward_dev(delta, bp, cp, x, rates, c1, y1, off, full, lanes * T, d, s)
    c2 = torch.zeros(lanes, d * s, device="cuda")
    y2 = torch.zeros(lanes * T, d, device="cuda")
    gpu.ssm_forward_dev(delta, bp, cp, x, rates, c2, y2, off, half, lanes * T, d, s)
    gpu.ssm_forward_dev(delta, bp, cp, x, rates, c2, y2, off + T // 2, half, lanes * T, d, s)
    torch.cuda.synchronize()
    gpu.set_stream(None)
    assert torch.equal(y1, y2) and torch.equal(c1, c2)
    assert bool(torch.isfinite(y1).all())


def test_shape_and_lane_errors(gpu):
    import pssa_b200
    delta, bp, cp, x, rates, h0 = inputs(4, 8, 4, 0)
    y = np.full((4, 8), 7.0, np.float32)
    with pytest.raises(pssa_b200.B200Error) as e:
        gpu.ssm_forward(delta[:3], bp, x, rates, cp, h0, 4, 8, 4, y_ssm=y)
    assert e.value.status == 2 and "shape mismatch" in str(e.value) and np.all(y == 7.0)
    with pytest.raises(pssa_b200.B200Error) as e:
        gpu.ssm_forward(delta[:0], bp[:0], x[:0], rates, cp[:0], h0, 0, 8, 4, y_ssm=y[:0])
    assert "must be positive" in str(e.value)
    import torch
    z = torch.zeros(4, 8, device="cuda")
    with pytest.raises(pssa_b200.B200Error) as e:
        gpu.ssm_forward_dev(z, z, z, z, z, None, z, np.array([0, 3], np.uint32), np.array([3, 2], np.uint32), 4, 8, 4)
    assert e.value.status == 2 and "outside 4 rows" in str(e.value)


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("s", [48, 64, 32, 16])
def test_edge_values_of_the_decay_reach_every_state(gpu, s, exact):
    """Rates and deltas outside the model's (a NaN, infinities, positive rates up to and past overflow), in the states whose exponential
    is the polynomial (0 and 1 of every 16 in the kernel that 48 states take) and in their neighbours, and in the few-lanes kernel
    (16, 32, 64 states), whose tiles are padded with tokens of delta 0. There an infinite rate at a delta of 0 leaves a state as it
    is, elsewhere it is a NaN: that one pair is left out."""
    import torch
    d, T = 64, 2
    rng = np.random.default_rng(4)
    rates = -rng.uniform(0.01, 0.7, (d, s)).astype(np.float32)
    delta = np.full((T, d), 1.0, np.float32)
    delta[1] = 0.5
    edge = [np.nan, np.inf, -np.inf, 88.5, 89.5, 127.0, 200.0, 1e30, -1e30, 0.5, 0.0, -87.0, -103.0]
    for i, v in enumerate(edge):
        rates[i, [0, 1, 2, 3, s // 3, s // 3 + 1, s - 1]] = v
    delta[0, 20], delta[0, 21], delta[0, 22], delta[0, 23] = np.nan, 0.0, -200.0, np.inf
    rates[21, [0, 5]], rates[23, [0, 5]] = np.inf if s == 48 else 0.1, 0.0
    b, c = rng.normal(0, 1, (T, s)).astype(np.float32), rng.normal(0, 1, (T, s)).astype(np.float32)
    x, h0 = rng.normal(0, 1, (T, d)).astype(np.float32), rng.normal(0, 1, (d, s)).astype(np.float32)
    want = h0.astype(np.float64)
    size = np.abs(want)  # of the terms: they can cancel
    with np.errstate(all="ignore"):
        for t in range(T):
            a = np.exp((delta[t][:, None].astype(np.float64) * rates)).astype(np.float32).astype(np.float64)
            u = (delta[t] * x[t]).astype(np.float64)[:, None] * b[t]
            want, size = a * want + u, a * size + np.abs(u)
            want = want.astype(np.float32).astype(np.float64)
    carry = torch.from_numpy(h0.copy()).cuda()
    y = torch.zeros(T, d, device="cuda")
    dev = [torch.from_numpy(v).cuda() for v in (delta, b, c, x, rates)]
    torch.cuda.synchronize()
    gpu.ssm_forward_dev(*dev, carry, y, None, None, T, d, s, exact=exact)
    gpu.synchronize()
    got = carry.cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isinf(got), np.isinf(want))
    fin = np.isfinite(want)
    assert np.array_equal(np.sign(got[np.isinf(want)]), np.sign(want[np.isinf(want)]))
    # the argument carries three roundings of 2^-24 of at most 128, the exponential 2^-22; below 2^-126 a decay may stay there
    assert np.max(np.abs(got[fin] - want[fin]) / np.maximum(size[fin], 1e-30)) <= 2 * (3 * 128 * 2.0 ** -24 + 2.0 ** -22)  # two tokens
    with np.errstate(all="ignore"):
        assert np.array_equal(np.isnan(y.cpu().numpy()[1]), np.isnan((want * c[1]).sum(1)))


# two channels a thread, 352 and 256 threads a CTA (one, 16 and 48 lanes of up to 768 channels); tiles of 32 tokens and a tail; the last states
# of a thread whole, in part, and those of a width that shorter calls take to another kernel
@pytest.mark.parametrize("lanes,d,s,T", [(1, 68, 60, 261), (16, 768, 52, 256), (48, 768, 60, 291), (48, 768, 64, 263)])
def test_small_argument_tiles_and_their_borders(gpu, lanes, d, s, T):
    """Calls of 256 tokens a lane or more, whose tiles take the polynomial of small arguments for states 48 to 63 where a warp's exponents
    allow it: rates of zero and at the limit (channels 4 and 5), of the other sign and NaN (20 and 36, whose warps never take
    it), and a delta at, past and far past the limit, negative, infinite and NaN (50 to 55), each in a tile of its own between
    tiles that do. The same tokens in two shorter calls, which never take it, give other bits exactly there."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(d + s)
    f = lambda *sh: torch.randn(*sh, device="cuda", generator=g)  # noqa: E731
    rows = lanes * T
    delta = torch.rand(rows, d, device="cuda", generator=g)
    rates = -torch.exp(torch.empty(d, s, device="cuda").uniform_(-5.0, -1.4, generator=g))  # all below 0.4 / log2(e) = 0.277
    rates[4, 50], rates[5, 49], rates[20, 50], rates[36, 49], rates[50, 48:] = 0.0, -0.277, 0.02, float("nan"), -0.25
    special = ((1, 50, 0.4 / 1.4427 / 0.25), (2, 50, 0.401 / 1.4427 / 0.25), (3, 51, 3.0), (4, 52, -1.0), (5, 53, float("inf")), (6, 54, float("nan")), (7, 55, 60.0))
    for tile, ch, v in special:
        delta[tile * 32 + tile, ch] = v
    bp, cp, x, h0 = f(rows, s), f(rows, s), f(rows, d), f(lanes, d * s)
    carry, y, carry2, y2 = h0.clone(), torch.zeros(rows, d, device="cuda"), h0.clone(), torch.zeros(rows, d, device="cuda")
    off = np.arange(lanes) * T
    gpu.set_stream(torch.cuda.current_stream())
    for c, out, parts in ((carry, y, ((0, T),)), (carry2, y2, ((0, 128), (128, T - 128)))):
        for t0, n in parts:
            gpu.ssm_forward_dev(delta, bp, cp, x, rates, c, out, (off + t0).astype(np.uint32), np.full(lanes, n, np.uint32), rows, d, s)
    torch.cuda.synchronize()
    gpu.set_stream(None)
    if s != 64:  # (64 states: the two shorter calls are the few-lanes kernel's)
        a, b = (v.reshape(lanes, d, s).view(torch.int32) for v in (carry, carry2))
        assert not torch.equal(a[:, :8, 48:], b[:, :8, 48:])
        never = [ch for ch in list(range(16, 24)) + list(range(32, 40)) if ch != 36]
        assert torch.equal(a[:, never], b[:, never])
    q = lambda a, w: a.double().reshape(lanes, T, w)  # noqa: E731
    dl, b, c, xv, want = q(delta, d), q(bp, s), q(cp, s), q(x, d), h0.double().reshape(lanes, d, s)
    size = want.abs()  # of the terms: they can cancel
    for i in range(T):
        a = torch.exp(dl[:, i, :, None] * rates.double())
        u = (dl[:, i] * xv[:, i])[:, :, None] * b[:, i, None, :]
        want, size = a * want + u, a * size + u.abs()
        got, ref, mag = q(y, d)[:, i], (want * c[:, i, None, :]).sum(2), (size * c[:, i, None, :].abs()).sum(2)
        assert torch.equal(torch.isnan(got), torch.isnan(ref))
        # a token: the argument's two roundings (2^-24 of at most 60 * 0.25 / ln 2 = 22) and the exponential's 2^-22; sums 2^-24 each
        fin = torch.isfinite(ref)
        assert float(((got - ref).abs() / mag)[fin].max()) <= (i + 1) * 2.0 ** -22 + (2 * 22 + s) * 2.0 ** -24
    got = carry.double().reshape(lanes, d, s)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    fin = torch.isfinite(want)
    assert float(((got - want).abs() / size)[fin].max()) <= T * 2.0 ** -22 + 2 * 22 * 2.0 ** -24
