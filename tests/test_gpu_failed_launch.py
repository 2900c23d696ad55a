"""A launch that fails half-way through a call: the error is told, and the same call made again gives the results of an
undisturbed run. The failure is made on the host (es_fail_launch tells a launch that ran as failed); the counts that a
step's last kernels would have left clear are then what the next one must not add to."""

import ctypes

import numpy as np
import pytest

import es_b200
import es_synth
from gpu_util import to_dev
from test_gpu_cambi import banded

pytestmark = pytest.mark.gpu

CAMBI_LAUNCHES = 6


def fails(n, call):
    es_b200.fail_launch(n)
    try:
        with pytest.raises(es_b200.EsError) as e:
            call()
    finally:
        es_b200.fail_launch(0)
    assert e.value.status == es_b200.ES_ERR_CUDA


def test_cambi_after_each_failed_launch(cuda, module):
    w, h = 256, 192
    pictures = [banded(w, h, 3 + k, step=2) for k in range(2)]
    planes = [to_dev(cuda, p) for p in pictures]
    stream = cuda.cuda.current_stream().cuda_stream
    params = es_b200.derive_params(w, h)
    params.topk = 0.3

    def run(c, k):
        c.launch(planes[k].data_ptr(), w, stream)
        return c.finish(), c.scale_stats()

    clean = es_b200.Cambi(module, w, h, 10, params)
    before = es_b200.launch_count()
    want = [run(clean, k) for k in range(2)]
    assert es_b200.launch_count() - before == 2 * CAMBI_LAUNCHES
    clean.close()
    assert all(counts[0] > 0.3 * w * h for _, (_, _, counts) in want)  # the selection runs
    for n in range(1, CAMBI_LAUNCHES + 1):
        c = es_b200.Cambi(module, w, h, 10, params)
        fails(n, lambda: c.launch(planes[0].data_ptr(), w, stream))
        assert [run(c, k) for k in (1, 0, 1)] == [want[1], want[0], want[1]], n
        c.close()


def steps_of(torch, w, h, count):
    """Banded sources and encodes (most pixels have a c-value: the selection runs) with some grain in a corner (structure
    and lasting texture), as device frames."""
    rng = np.random.default_rng(8)
    grain = np.zeros((h, w))
    grain[: h // 2, : w // 3] = rng.normal(0, 12, (h // 2, w // 3))
    out = []
    for f in range(count):
        src = np.clip(banded(w, h, 5, step=2) + np.rint(grain), 0, 1023).astype(np.uint16)
        encs = [np.clip(banded(w, h, 5 + e, step=2) + np.rint(grain * (0.7 - 0.2 * e)) + (f % 2), 0, 1023).astype(np.uint16) for e in range(2)]
        pic = [es_synth.Picture(y, *(2 * [es_synth._chroma(y)]), 10) for y in [src] + encs]
        out.append(es_b200.device_step(torch, es_synth.Step(pic[0], pic[1:])))
    return out


@pytest.mark.parametrize("form", ["frame", "batch", "batch without graphs"])
def test_frame_steps_after_each_failed_launch(cuda, module, form):
    w, h, frames = 192, 128, 19
    stream = cuda.cuda.current_stream().cuda_stream
    steps = steps_of(cuda, w, h, frames)

    def run(fail_at):
        if form == "frame":
            sc = es_b200.Frame(module, w, h, 10, 2)
            queue = lambda f: sc.queue(f, steps[f][1][0], steps[f][1][1:], stream)
        else:
            sc = es_b200.Batch(module, [(w, h, 10, 2)], use_graphs=form == "batch")
            queue = lambda f: sc.queue(f, steps[f][1], stream)
        accs = [es_b200.new_accum() for _ in range(2)]
        results, launches = [], []
        for f in range(frames):
            if f in fail_at:  # with the step before it not yet collected
                fails(fail_at[f], lambda: queue(f))
            before = es_b200.launch_count()
            queue(f)
            launches.append(es_b200.launch_count() - before)
            if f:
                results += sc.collect(f - 1, accs, accs)
        results += sc.collect(frames - 1, accs, accs)
        sc.close()
        return [bytes(r) for r in results], [ctypes.string_at(ctypes.addressof(a), ctypes.sizeof(a)) for a in accs], launches

    want = run({})
    assert want[2][1] >= 13 and want[2][13] >= 14
    # a launch of each step fails in turn: every one of the steps without the lasting texture, and of those with it
    got = run({f: f for f in range(1, 14)})
    assert got[:2] == want[:2]
    got = run({f: 1 + (f * 5) % 14 for f in range(12, frames)})
    assert got[:2] == want[:2]
