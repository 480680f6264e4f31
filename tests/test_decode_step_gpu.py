"""A decode step as one kernel (step_decode.cu): tile edges of its row counts, and one order of every sum whatever the batch."""
import numpy as np
import pytest

import oracle as O
from helpers import fill_synthetic, upload
from parity import scale_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import pssa_b200
    d = pssa_b200.B200Dispatch(0)
    yield d
    d.close()


def models(gpu, depth, v, d, s, cap, fill, streams):
    import pssa_b200
    om = O.Model.new(depth, v, d, s, 64, cap, tau_mem=0.1, seed=d + s)
    fill_synthetic(om, d + s, fill)
    out = []
    for precision in (0, 1):
        m = pssa_b200.PSSAModel(gpu, depth, v, d, s, 64, cap, tau_mem=0.1, streams=streams, precision=precision)
        upload(om, m)
        out.append(m)
    return out


# widths whose products end inside a tile, every state width, a partly filled bank, a vocabulary that is no tile's multiple
@pytest.mark.parametrize("depth,v,d,s,cap,fill", [(2, 301, 96, 16, 128, 0.7), (2, 513, 192, 64, 512, 1.0), (3, 97, 160, 32, 64, 1.0)])
def test_every_tile_edge_of_the_rows(gpu, depth, v, d, s, cap, fill):
    big, exact = models(gpu, depth, v, d, s, cap, fill, 130)
    rng = np.random.default_rng(1)
    prompts = [rng.integers(1, v, 40) for _ in range(130)]
    for m in (big, exact):
        m.prefill_batch(prompts, want_logits=False)
    ids = rng.integers(1, v, 130)
    state = {m: [m.copy_recurrent_state_to(i) for i in range(130)] for m in (big, exact)}
    want = exact.decode_step(ids)
    full = big.decode_step(ids[:128])
    assert scale_err(full, want[:128]) <= 2e-2
    after = big.copy_recurrent_state_to(127)
    for n in (1, 7, 8, 9, 16, 17, 32, 33, 63, 64, 65, 127):
        pick = rng.permutation(128)[:n].astype(np.uint32)  # any streams, in any order
        for i in pick:
            big.copy_recurrent_state_from(state[big][i], int(i))
        got = big.decode_step(ids[pick], pick)
        assert np.array_equal(got, full[pick]), n  # the same bits alone and in a batch
    big.copy_recurrent_state_from(state[big][127], 127)
    big.decode_step(ids[127:128], [127])
    assert np.array_equal(big.copy_recurrent_state_to(127), after)
    for i in range(130):
        big.copy_recurrent_state_from(state[big][i], i)
    assert scale_err(big.decode_step(ids), want) <= 2e-2  # above the kernel's rows: the block schedule
    big.close(), exact.close()
