"""The text of a wait that ran out names no one kind of wait: a strip copy, a
neighbour's rows, their readers and the team's lock share the status."""
import pytest

from gpu_util import make_classifier, reads_of_lengths, small_genome
from dtwax_gb300 import synth

pytestmark = pytest.mark.gpu


def test_timeout_text_is_of_any_bounded_wait(built_lib):
    import dtwax_gb300 as d
    g, tab = small_genome(20_000, 91), synth.level_table()
    reads = reads_of_lengths(g, g, tab, [300, 200])
    with make_classifier(g, tab, precision=d.FP16) as clf:
        clf.debug_stall_next(0, 4096)
        with pytest.raises(d.DtwxError) as e:
            clf.classify(raw=reads.raw, offsets=reads.offsets)
    assert e.value.code == -6
    assert "bounded wait gave up" in str(e.value) and "TMA" not in str(e.value)
