"""Replays of a captured device batch (use_graphs) between other calls on the handle.

A captured graph holds the addresses of the handle's scratch buffers and a
launch shape.  A call that makes a buffer grow frees the old one, and a tuned
shape is to be used from then on, so after either the batch runs directly
again, is captured again and then replayed; every run gives the same results.
A call that changes neither leaves the graph as it is.
"""
import numpy as np
import pytest

from gpu_util import make_classifier, reads_of_lengths, small_genome
from dtwax_gb300 import synth

pytestmark = pytest.mark.gpu

LENGTHS = [700, 1200, 33]
MORE = [2000, 4000] * 60  # every buffer of such a call is larger than of LENGTHS


@pytest.fixture(scope="module")
def case(built_lib):
    g, o = small_genome(30_000, 51), small_genome(30_000, 52)
    tab = synth.level_table()
    return g, tab, reads_of_lengths(g, o, tab, LENGTHS), reads_of_lengths(g, o, tab, MORE)


def between(clf, kind, few, more, stream):
    import torch
    raw = torch.tensor(more.raw, device="cuda")
    out = torch.zeros(32 * more.n, dtype=torch.uint8, device="cuda")
    if kind == "classify":
        clf.classify(raw=more.raw, offsets=more.offsets)
    elif kind == "classify_device":
        clf.classify_device(raw.data_ptr(), more.offsets, out.data_ptr(), stream.cuda_stream)
    elif kind == "distances":
        clf.distances(raw.data_ptr(), more.offsets, out.data_ptr(), stream.cuda_stream)
    elif kind == "normalize":
        clf.normalize(raw.data_ptr(), more.offsets, torch.empty_like(raw).data_ptr(), stream.cuda_stream)
    elif kind == "autotune":
        clf.autotune(len(LENGTHS), int(np.mean(LENGTHS)))
    else:
        clf.classify(raw=few.raw, offsets=few.offsets)  # nothing grows
    torch.cuda.synchronize()


@pytest.mark.parametrize("kind", ["classify", "classify_device", "distances", "normalize", "autotune", "small"])
def test_a_graph_ends_with_the_buffers_it_holds(case, kind):
    import torch
    import dtwax_gb300 as d
    g, tab, few, more = case
    with make_classifier(g, tab, precision=d.FP32, use_graphs=1) as clf:
        stream = torch.cuda.Stream()
        raw = torch.tensor(few.raw, device="cuda")
        out = torch.zeros(32 * few.n, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

        def run():
            out.zero_()
            torch.cuda.synchronize()
            clf.classify_device(raw.data_ptr(), few.offsets, out.data_ptr(), stream.cuda_stream)
            stream.synchronize()
            return np.frombuffer(out.cpu().numpy().tobytes(), d.RESULT_DTYPE).copy(), clf.tuning()["graph_replays"]

        want, replays = run()
        assert replays == 0
        seen = [run() for _ in range(2)]
        assert [n for _, n in seen] == [0, 1]  # captured, replayed
        between(clf, kind, few, more, stream)
        after = [run() for _ in range(3)]
        # the graph is gone: a direct run, a capture, a replay (or it was kept, and replays)
        assert [n for _, n in after] == ([2, 3, 4] if kind == "small" else [1, 1, 2])
    for got, _ in seen + after:
        for k in ("score_fwd", "score_rev", "end_pos", "strand", "call"):
            np.testing.assert_array_equal(got[k], want[k], err_msg=k)  # FP32: the same bits for every shape


def test_sync_waits_for_a_replay(built_lib):
    """dtwx_sync returns once the replayed kernels are through, as after a
    direct call (the batch takes a few milliseconds)."""
    import torch
    import dtwax_gb300 as d
    g = small_genome(200_000, 53)
    tab = synth.level_table()
    reads = reads_of_lengths(g, g, tab, [2000] * 200)
    with make_classifier(g, tab, precision=d.FP16, use_graphs=1) as clf:
        stream = torch.cuda.Stream()
        raw = torch.tensor(reads.raw, device="cuda")
        out = torch.zeros(32 * reads.n, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        for replays in (0, 0, 1, 2):
            clf.classify_device(raw.data_ptr(), reads.offsets, out.data_ptr(), stream.cuda_stream)
            clf.sync()
            assert stream.query()
            assert clf.tuning()["graph_replays"] == replays
