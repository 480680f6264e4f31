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
