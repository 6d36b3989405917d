"""PIC steps of one size from several streams and threads.

Calls with the same device, particle count and resolution share a solver, so
they have to run one after another on the device.  Bound: two runs of one step
differ by FP32 summation order; a node sums at most a few hundred particles'
terms, 1e-5 of a field's largest value."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, RES, ROUNDS = 60000, 48, 20


def _inputs(torch, seed):
    rng = np.random.default_rng(seed)
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device="cuda")
    leaf = [t(rng.uniform(0.1, 0.9, (N, 3))), t(rng.normal(0, 1, (N, 3))), t(rng.uniform(0.5, 1.5, N)),
            t([0.1 * seed, -9.8 + seed, 0.3])]
    for a in leaf:
        a.requires_grad_(True)
    return leaf, [t(rng.normal(0, 1, (N, 3))), t(rng.normal(0, 1, (N, 3)))]


def _pass(torch, leaf, go, dt):
    from physgrad_b200.autograd import MPMTimestep

    xo, vo = MPMTimestep.apply(*leaf, RES, dt)
    return [xo.detach(), vo.detach(), *torch.autograd.grad([xo, vo], leaf, go)]


def _agree(got, want):
    for a, b in zip(got, want):
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())


@pytest.mark.parametrize("dts", [(1e-3, 1e-3, 1e-3), (1e-3, 2e-3, 5e-4)])
@pytest.mark.parametrize("threads", [False, True])
def test_steps_of_one_size_on_several_streams(gpu, threads, dts):
    import torch

    data = [_inputs(torch, k) for k in range(len(dts))]
    want = [_pass(torch, *d, dt) for d, dt in zip(data, dts)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in dts]
    got = [[] for _ in dts]

    def turn(k):
        with torch.cuda.stream(streams[k]):
            got[k].append(_pass(torch, *data[k], dts[k]))

    if threads:
        ts = [threading.Thread(target=lambda k=k: [turn(k) for _ in range(ROUNDS)]) for k in range(len(dts))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for _ in range(ROUNDS):
            for k in range(len(dts)):
                turn(k)
    torch.cuda.synchronize()
    for k in range(len(dts)):
        assert len(got[k]) == ROUNDS
        for g in got[k]:
            _agree(g, want[k])
    _agree(_pass(torch, *data[0], dts[0]), want[0])  # and the solver is sound afterwards
