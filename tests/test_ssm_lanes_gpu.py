"""The few-lanes split of the fused SSM stage (ssm_fused.cu): its lane splits, tile tails and channel tails against the oracle."""
import numpy as np
import pytest

import oracle as O
from parity import REL_TOL, chan_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import pssa_b200
    d = pssa_b200.B200Dispatch(0)
    yield d
    d.close()


# lengths around the 16- and 32-token tiles, one call per lane split: (channels in flight) x (states)
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("d,s,lengths", [(20, 64, [64]), (772, 64, [65, 1]), (768, 64, [130, 0, 97, 64, 64, 64]), (36, 32, [66]),
                                         (388, 32, [80] * 6), (12, 16, [95]), (196, 16, [64] * 24), (192, 64, [7, 16, 17, 33])])
def test_few_lanes_matches_the_ordered_recurrence(gpu, d, s, lengths, exact):
    import torch
    rng = np.random.default_rng(d + s)
    lengths = np.array(lengths, np.uint32)
    offsets = np.concatenate([[0], np.cumsum(lengths)[:-1]]).astype(np.uint32)
    rows, n = int(lengths.sum()), len(lengths)
    f = lambda *sh: rng.normal(0, 1, sh).astype(np.float32)  # noqa: E731
    delta = np.log1p(np.exp(f(rows, d))).astype(np.float32)
    bp, cp, x, carry = f(rows, s), f(rows, s), f(rows, d), f(n, d * s)
    rates = -np.exp(rng.uniform(np.log(0.005), np.log(0.7), d * s)).astype(np.float32)
    ref_carry = carry.copy()
    ref_y = O.ssm_lanes(delta, bp, cp, x, rates, ref_carry, offsets, lengths)
    t = [torch.from_numpy(v).cuda() for v in (delta, bp, cp, x, rates, carry)]
    y, states = torch.zeros(rows, d, device="cuda"), torch.zeros(rows, d * s, device="cuda")
    y2, c2 = torch.zeros_like(y), t[5].clone()
    gpu.set_stream(torch.cuda.current_stream())
    gpu.ssm_forward_dev(*t, y, offsets, lengths, rows, d, s, exact=exact)
    gpu.ssm_forward_dev(*t[:5], c2, y2, offsets, lengths, rows, d, s, states=states, exact=exact)
    torch.cuda.synchronize()
    tol = 5e-6 if exact else REL_TOL
    assert chan_err(y.cpu().numpy(), ref_y, 0) <= tol
    for off, ln in zip(offsets, lengths):
        if ln:  # the tape's last row is the carry out
            assert torch.equal(states[off + ln - 1], c2[[i for i in range(n) if offsets[i] == off and lengths[i]][0]])
    assert chan_err(t[5].cpu().numpy().ravel(), ref_carry.ravel(), 0) <= tol
    assert torch.equal(c2, t[5])
    if exact:
        assert torch.equal(y, y2)


def test_eight_lanes_of_a_wide_model_take_the_eight_by_eight_split(gpu):
    """The split chosen where a sixth CTA of the 16 x 4 one would not fit an SM, against the recurrence in f64 (tile tails included)."""
    import torch
    lanes, T, d, s = 8, 277, 768, 64
    g = torch.Generator(device="cuda").manual_seed(2)
    f = lambda *sh: torch.randn(*sh, device="cuda", generator=g)  # noqa: E731
    delta = torch.nn.functional.softplus(f(lanes * T, d)).contiguous()
    rates = -torch.exp(torch.empty(d, s, device="cuda").uniform_(-5.0, -0.4, generator=g))
    bp, cp, x, carry = f(lanes * T, s), f(lanes * T, s), f(lanes * T, d), f(lanes, d * s)
    h = carry.double().reshape(lanes, d, s)
    off, ln = (np.arange(lanes) * T).astype(np.uint32), np.full(lanes, T, np.uint32)
    y = torch.zeros(lanes * T, d, device="cuda")
    gpu.set_stream(torch.cuda.current_stream())
    gpu.ssm_forward_dev(delta, bp, cp, x, rates, carry, y, off, ln, lanes * T, d, s)
    torch.cuda.synchronize()
    gpu.set_stream(None)
    q = lambda a: a.double().reshape(lanes, T, -1)  # noqa: E731
    dl, b, c, xv = q(delta), q(bp), q(cp), q(x)
    want = []
    for t in range(T):
        h = torch.exp(dl[:, t, :, None] * rates.double()) * h + (dl[:, t] * xv[:, t])[:, :, None] * b[:, t, None, :]
        want.append((h * c[:, t, None, :]).sum(2))
    assert chan_err(y.cpu().numpy(), torch.stack(want, 1).reshape(lanes * T, d).cpu().numpy(), 0) <= REL_TOL
    assert chan_err(carry.cpu().numpy().ravel(), h.cpu().numpy().ravel(), 0) <= REL_TOL
