"""Read Until batches whose work items are shared out to the CTAs in advance.

A chunk of the reference may only overwrite its saved row once the chunks to
its right have read theirs, so items wait for items of lower number.  Several
items per CTA is where an order of the CTAs would matter: results have the bits
of single warps that take the items one after the other, and a batch ends while
another kernel holds most of the GPU, that is, with CTAs that have not started.
"""
import time

import numpy as np
import pytest

from gpu_util import make_classifier, reads_of_lengths, small_genome
from dtwax_gb300 import synth

pytestmark = pytest.mark.gpu

CHUNK = 1600


def serve(clf, raw, reads, first=1):
    """Three chunks of every read; {(read, chunks): (score, end, strand)} and the shape."""
    for k in range(3):
        for r in range(reads):
            clf.submit_chunk(r, first + r, raw[CHUNK * k:CHUNK * (k + 1)], is_last=k == 2)
        clf.serve_step()
        clf.serve_drain()
    got = clf.poll_decisions(4096)
    return {(d["read_number"] - first, d["chunks"]): (d["score"], d["end_pos"], d["strand"]) for d in got}


@pytest.mark.parametrize("precision,state,reads,genome", [
    (0, 0, 1, 500_000), (0, 1, 1, 500_000), (0, 0, 16, 50_000), (0, 1, 15, 50_000), (0, 0, 2, 70_000),
    (1, 0, 16, 50_000), (1, 0, 3, 60_000), (2, 0, 16, 50_000), (2, 0, 3, 60_000)])
def test_dealt_rows_have_the_bits_of_single_warps(built_lib, precision, state, reads, genome):
    g, tab = small_genome(genome, 61), synth.level_table()
    raw = reads_of_lengths(g, g, tab, [3 * CHUNK]).raw
    cfg = dict(precision=precision, state_precision=state, threshold=-1.0)
    with make_classifier(g, tab, **cfg) as clf:
        clf.serve_start(max_in_flight=reads, chunks_per_decision=3)
        got = serve(clf, raw, reads)
        shape = clf.tuning()
    assert shape["dealt"] == 1
    if reads in (1, 15, 16):
        assert shape["work_items"] > shape["ctas"]  # several items to a CTA
    with make_classifier(g, tab, warps_per_cta=1, cells_per_thread=shape["cells_per_thread"],
                         chunk_strips=shape["chunk_strips"], **cfg) as clf:
        clf.serve_start(max_in_flight=reads, chunks_per_decision=3)
        want = serve(clf, raw, reads)
        assert clf.tuning()["dealt"] == 0
    assert got == want and len(got) == 3 * reads
    assert len({got[r, 3] for r in range(reads)}) == 1  # every read is the same read


def test_dealt_rows_end_while_another_kernel_holds_the_gpu(built_lib):
    """All SMs but one are held for about a second by a batch of another handle
    (16-warp CTAs, all the registers of an SM); one read is served on the last."""
    import torch
    import dtwax_gb300 as d
    tab = synth.level_table()
    big, g = small_genome(1_000_000, 62), small_genome(500_000, 63)
    raw = reads_of_lengths(g, g, tab, [3 * CHUNK]).raw
    with make_classifier(g, tab, precision=d.FP16, threshold=-1.0) as clf, \
            make_classifier(big, tab, precision=d.FP16, recurrence=d.REF_DEL, warps_per_cta=16) as other:
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        clf.serve_start(max_in_flight=1, chunks_per_decision=3)
        want = serve(clf, raw, 1)
        shape = clf.tuning()
        assert shape["dealt"] == 1 and shape["work_items"] > shape["ctas"] == sms
        held = reads_of_lengths(big, big, tab, [2400])
        n = 16 * (sms - 1)
        x = torch.tensor(np.tile(held.raw, n), device="cuda")
        out = torch.zeros(32 * n, dtype=torch.uint8, device="cuda")
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        other.classify_device(x.data_ptr(), 2400 * np.arange(n + 1, dtype=np.int64), out.data_ptr(),
                              stream.cuda_stream)
        time.sleep(0.05)
        t = time.perf_counter()
        got = serve(clf, raw, 1, first=11)
        took = (time.perf_counter() - t) * 1e3
        other.sync()
        assert other.tuning()["ctas"] == sms - 1
        assert took < other.last_sweep_ms() / 2  # not behind the other batch (about 135 ms of 835)
        assert got == want
