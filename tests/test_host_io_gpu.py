"""Host arrays in and out of the entry points (host_io.cu): several windows of the pinned buffer, pieces that straddle arrays, threads."""
import threading
import time

import numpy as np
import pytest

import oracle as O
from parity import chan_err

pytestmark = pytest.mark.gpu


def ssm_inputs(T, d, s, seed):
    rng = np.random.default_rng(seed)
    delta = rng.uniform(0.01, 0.3, (T, d)).astype(np.float32)
    b, c, x = (rng.standard_normal((T, n)).astype(np.float32) for n in (s, s, d))
    return delta, b, c, x, -rng.uniform(0.01, 0.7, d * s).astype(np.float32), rng.standard_normal(d * s).astype(np.float32)


def host_call(gpu, T, d, s, inp):
    """All four outputs of one call, in memory that nothing has touched before."""
    delta, b, c, x, rates, h0 = inp
    states, bar_a, bar_b, y = (np.full(n, np.nan, np.float32) for n in ((T + 1) * d * s, T * d * s, T * d * s, T * d))
    gpu.ssm_forward(delta, b, x, rates, c, h0, T, d, s, bar_a, bar_b, states, y)
    return states, bar_a, bar_b, y


def device_call(gpu, T, d, s, inp):
    import torch
    delta, b, c, x, rates, h0 = (torch.from_numpy(v).cuda() for v in inp)
    y = torch.zeros(T * d, device="cuda")
    states, bar_a, bar_b = (torch.zeros(T * d * s, device="cuda") for _ in range(3))
    torch.cuda.synchronize()
    gpu.ssm_forward_dev(delta, b, c, x, rates, h0, y, None, None, T, d, s, states, bar_a, bar_b)
    gpu.synchronize()
    return np.concatenate([inp[5], states.cpu().numpy()]), bar_a.cpu().numpy(), bar_b.cpu().numpy(), y.cpu().numpy()


# outputs below the threads' size, of a window and a bit, of several windows; widths whose arrays end inside a piece and a share
@pytest.mark.parametrize("T,d,s", [(5, 7, 3), (257, 36, 16), (701, 37, 13), (1031, 64, 16), (1500, 61, 32)])
def test_outputs_of_a_call_arrive_whole_whatever_their_size(T, d, s):
    import pssa_b200
    gpu = pssa_b200.B200Dispatch(0)
    inp = ssm_inputs(T, d, s, T)
    want = device_call(gpu, T, d, s, inp)
    for _ in range(2):  # the second one finds the kept buffers
        got = host_call(gpu, T, d, s, inp)
        for g, w in zip(got, want):
            assert np.array_equal(g, w)
    ref = O.ssm_forward(inp[0], inp[1], inp[2], inp[3], inp[4], inp[5], mode=0)
    assert chan_err(got[3].reshape(T, d), ref[1], 0) <= 1e-5
    gpu.close()


def test_contexts_in_several_threads_and_closed_ones():
    """Contexts in three threads at once, of which one at a time has the copying threads, closed and opened again in between: a new
    one takes over the pinned buffer of one that is gone."""
    import pssa_b200
    T, d, s = 900, 61, 32
    failures = []

    def work(k):
        try:
            inp = ssm_inputs(T + k, d, s, k)
            for _ in range(3):
                gpu = pssa_b200.B200Dispatch(0)
                want = device_call(gpu, T + k, d, s, inp)
                for _ in range(4):
                    for g, w in zip(host_call(gpu, T + k, d, s, inp), want):
                        assert np.array_equal(g, w)
                gpu.close()
        except BaseException as e:  # noqa: B036
            failures.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_one_thread_waits_for_the_kernels_in_front_of_a_large_output():
    """A long piece of work on the stream before the outputs: the process spends one core's time on the wait, not that of the
    copying threads too."""
    import pssa_b200
    import torch
    gpu = pssa_b200.B200Dispatch(0, torch.cuda.current_stream())
    T, d, s = 900, 61, 32
    inp = ssm_inputs(T, d, s, 1)
    host_call(gpu, T, d, s, inp)
    torch.cuda._sleep(600_000_000)  # about 0.3 s of the device's clock
    wall, cpu = time.perf_counter(), time.process_time()
    host_call(gpu, T, d, s, inp)
    wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
    gpu.close()
    assert wall > 0.15
    assert cpu <= 1.5 * wall, (cpu, wall)


@pytest.mark.parametrize("vocab,lanes", [(16384, 4), (16384, 5), (16384, 17), (4099, 63), (4099, 130), (16384, 70)])
def test_logits_of_many_lanes_reach_their_places(vocab, lanes):
    """Logits that the first pinned buffer holds, that it does not hold (the driver's copy, and the largest buffer from the second call on)
    and of more than one window of that: a step of every lane and ragged calls with empty lanes between them, in a new context and
    again, equal the device-resident entry point's logits."""
    import torch
    import pssa_b200
    gpu = pssa_b200.B200Dispatch(0, torch.cuda.current_stream())
    d, s, k, cap = 32, 16, 64, 64
    m = pssa_b200.PSSAModel(gpu, 1, vocab, d, s, k, cap, tau_mem=0.1, streams=lanes, precision=0)
    m.init_random(5)
    rng = np.random.default_rng(lanes)
    keys = (rng.standard_normal((cap, k)) * 0.05).astype(np.float32)
    m.set_bank(0, keys, (keys ** 2).sum(1).astype(np.float32), rng.standard_normal((cap, d)).astype(np.float32), cap)
    for lengths in (np.ones(lanes, int), np.where(np.arange(lanes) % 5 == 2, 0, 1 + np.arange(lanes) % 3), np.arange(lanes) % 2):
        ids = [rng.integers(1, vocab, n) for n in lengths]
        flat = torch.from_numpy(np.concatenate(ids).astype(np.int32)).cuda()
        off = np.concatenate([[0], np.cumsum(lengths)[:-1]]).astype(np.uint32)
        want = torch.zeros(lanes, vocab, device="cuda")
        m.reset_recurrent_state()
        m.prefill_batch_dev(flat, off, lengths.astype(np.uint32), None, want)
        want = want.cpu().numpy()
        for _ in range(3):
            m.reset_recurrent_state()
            assert np.array_equal(m.prefill_batch(ids)[0], want)
    m.close()
    gpu.close()
