"""Separate handles driven by separate threads, with CTAs of different sizes.

The limit on a kernel's dynamic shared memory is a property of the function on
the device: a launch of 8-warp CTAs (53 KB) may not be refused because another
thread has just launched one-warp CTAs (7 KB) of the same kernel.
"""
import threading

import numpy as np
import pytest

from gpu_util import make_classifier, reads_of_lengths, small_genome
from dtwax_gb300 import synth

pytestmark = pytest.mark.gpu


def test_threads_do_not_take_shared_memory_from_each_other(built_lib):
    """One launch per read (dtwx_classify_plain_fp32), 200 reads a call, so that
    the threads' launches meet often."""
    g, tab = small_genome(6_000, 71), synth.level_table()
    reads = reads_of_lengths(g, g, tab, [40] * 200)
    failed, done = [], []
    go = threading.Barrier(4)

    def work(warps):
        try:
            with make_classifier(g, tab, precision=1, cells_per_thread=48, chunk_strips=64,
                                 warps_per_cta=warps) as clf:
                want = clf.classify(raw=reads.raw, offsets=reads.offsets)
                go.wait()
                for _ in range(60):
                    got = clf.classify_plain_fp32(raw=reads.raw, offsets=reads.offsets)
                    np.testing.assert_array_equal(got["score_fwd"], want["score_fwd"])
                done.append(warps)
        except Exception as e:  # (the barrier of the others must not wait for this thread)
            failed.append(e)
            go.abort()

    threads = [threading.Thread(target=work, args=(w,)) for w in (8, 1, 8, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed and len(done) == 4
