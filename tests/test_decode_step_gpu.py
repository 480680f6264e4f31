"""A decode step (step_decode.cu: one kernel, step_schedule.cu: a launch per stage): tile edges of its row counts, and one order of
every sum whatever the batch."""
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


def models(gpu, depth, v, d, s, k, cap, fill, streams):
    import pssa_b200
    om = O.Model.new(depth, v, d, s, k, cap, tau_mem=0.1, seed=d + s)
    fill_synthetic(om, d + s, fill)
    out = []
    for precision in (0, 1):
        m = pssa_b200.PSSAModel(gpu, depth, v, d, s, k, cap, tau_mem=0.1, streams=streams, precision=precision)
        upload(om, m)
        out.append(m)
    return out


# widths whose products end inside a tile, every state width, a partly filled bank, a vocabulary that is no tile's multiple; the
# widest model the step takes, with the wide keys and a bank too large to be staged
@pytest.mark.parametrize("depth,v,d,s,k,cap,fill", [(2, 301, 96, 16, 64, 128, 0.7), (2, 513, 192, 64, 64, 512, 1.0), (3, 97, 160, 32, 64, 64, 1.0),
                                                    (2, 130, 992, 64, 128, 1024, 0.9)])
def test_every_tile_edge_of_the_rows(gpu, depth, v, d, s, k, cap, fill):
    streams = 300
    big, exact = models(gpu, depth, v, d, s, k, cap, fill, streams)
    rng = np.random.default_rng(1)
    prompts = [rng.integers(1, v, 40) for _ in range(streams)]
    for m in (big, exact):
        m.prefill_batch(prompts, want_logits=False)
    ids = rng.integers(1, v, streams)
    state = [big.copy_recurrent_state_to(i) for i in range(streams)]
    want = exact.decode_step(ids)
    full = big.decode_step(ids)
    assert scale_err(full, want) <= 2e-2
    after = [big.copy_recurrent_state_to(i) for i in range(streams)]
    for n in (1, 7, 8, 9, 16, 17, 32, 33, 63, 64, 65, 127, 128, 129, 192, 255, 256, 257):
        pick = rng.permutation(streams)[:n].astype(np.uint32)  # any streams, in any order
        for i in pick:
            big.copy_recurrent_state_from(state[i], int(i))
        got = big.decode_step(ids[pick], pick)
        assert np.array_equal(got, full[pick]), n  # the same bits alone and in a batch
        assert all(np.array_equal(big.copy_recurrent_state_to(int(i)), after[i]) for i in pick[:3]), n
    big.close(), exact.close()


def test_idle_lanes_and_ids_in_any_place_do_not_change_a_stream(gpu):
    """Lanes without a token beside others, and (device entry) ids that lie apart and out of order: the logits and carries of the
    streams that do step are those of a batch of them alone; idle lanes keep theirs, and their rows of the result."""
    import torch
    v, streams = 301, 140
    big, exact = models(gpu, 2, v, 96, 16, 64, 128, 1.0, streams)
    rng = np.random.default_rng(2)
    big.prefill_batch([rng.integers(1, v, 24) for _ in range(streams)], want_logits=False)
    ids = rng.integers(1, v, streams)
    state = [big.copy_recurrent_state_to(i) for i in range(streams)]
    full = big.decode_step(ids)
    after = [big.copy_recurrent_state_to(i) for i in range(streams)]
    for live in ([0, 3, 4, 9], list(range(1, streams, 2)), list(range(0, streams - 1))):
        for i in range(streams):
            big.copy_recurrent_state_from(state[i], i)
        got = big.prefill_batch([ids[i:i + 1] if i in live else ids[:0] for i in range(streams)])[0]
        assert np.array_equal(got[live], full[live])
        for i in range(streams):
            assert np.array_equal(big.copy_recurrent_state_to(i), after[i] if i in live else state[i]), i
        for i in range(streams):
            big.copy_recurrent_state_from(state[i], i)
        place = rng.permutation(streams + 5)[:streams]
        held = np.zeros(streams + 5, np.int32)
        held[place] = ids
        lengths = np.array([i in live for i in range(streams)], np.uint32)
        logits = torch.full((streams, v), 7.0, device="cuda")
        greedy = torch.full((streams,), 7, device="cuda", dtype=torch.int32)
        torch.cuda.synchronize()  # the context has its own stream
        big.prefill_batch_dev(torch.from_numpy(held).cuda(), place.astype(np.uint32), lengths, None, logits, greedy)
        gpu.synchronize()
        got = logits.cpu().numpy()
        assert np.array_equal(got[live], full[live])
        idle = [i for i in range(streams) if i not in live]
        assert np.all(got[idle] == 7.0) and np.all(greedy.cpu().numpy()[idle] == 7)
        assert np.array_equal(greedy.cpu().numpy()[live], full[live][:, 1:].argmax(1) + 1)
        assert all(np.array_equal(big.copy_recurrent_state_to(i), after[i] if i in live else state[i]) for i in range(streams))
    big.close(), exact.close()


def test_more_rows_than_one_slice(gpu):
    v, streams = 65, 2050
    big, exact = models(gpu, 1, v, 32, 16, 64, 64, 1.0, streams)
    rng = np.random.default_rng(3)
    big.prefill_batch([rng.integers(1, v, 3) for _ in range(streams)], want_logits=False)
    ids = rng.integers(1, v, streams)
    state = [big.copy_recurrent_state_to(i) for i in (0, 2047, 2048, 2049)]
    full = big.decode_step(ids)
    for i, st in zip((0, 2047, 2048, 2049), state):
        big.copy_recurrent_state_from(st, i)
        assert np.array_equal(big.decode_step(ids[i:i + 1], [i])[0], full[i]), i
    big.close(), exact.close()


def test_steps_behind_a_prompt_and_after_reserve_allocate_nothing(gpu):
    """The step's scratch is part of the activation workspace: the first steps of a model that has read its prompts, and of a reserved
    one, leave the device's free memory as it is."""
    import pssa_b200
    import torch
    streams, d = 512, 768  # 12 MB of scratch: more than the allocator's granularity
    om = O.Model.new(1, 64, d, 16, 64, 64, tau_mem=0.1, seed=9)
    fill_synthetic(om, 9, 1.0)
    rng = np.random.default_rng(9)
    prompts = [rng.integers(1, 64, 2) for _ in range(streams)]
    ids = rng.integers(1, 64, streams)

    def model():
        m = pssa_b200.PSSAModel(gpu, 1, 64, d, 16, 64, 64, tau_mem=0.1, streams=streams, precision=0)
        upload(om, m)
        return m

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    first = model()  # loads the kernels, whose code takes memory too
    first.prefill_batch(prompts)
    want = first.decode_step(ids), first.decode_step(ids[:1], [0])
    read, reserved = model(), model()
    read.prefill_batch(prompts)
    reserved.reserve(2 * streams, streams)
    for m in (read, reserved):
        before = free()
        if m is reserved:
            m.decode_step(ids), m.decode_step(ids[:1], [0])
            m.reset_recurrent_state()
            m.prefill_batch(prompts)
        assert np.array_equal(m.decode_step(ids), want[0]) and np.array_equal(m.decode_step(ids[:1], [0]), want[1])
        assert free() == before
    first.close(), read.close(), reserved.close()
