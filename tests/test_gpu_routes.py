"""The launch routes that the bit-for-bit tests of the default shapes rely on.

Those tests compare results, whatever shape a batch got.  Here their batches,
and one more for FP32 path cost (whose teams of 4 they do not reach), have to
take every route between them: dealt items, single warps, teams of 4 and teams
of all warps of an SM.
"""
import pytest

import test_gpu_teams as teams
from gpu_util import make_classifier
from test_gpu_teams import batch, same_bits, setup  # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu

MIDDLE = [500] * 200  # reads between the lengths of single warps and of full teams


def params(test, name):
    return next(m.args[1] for m in test.pytestmark if m.name == "parametrize" and m.args[0] == name)


def routes(setup, precision, batches):
    g, _, tab = setup
    seen = {}
    for lengths in batches:
        reads = batch(setup, lengths)
        with make_classifier(g, tab, precision=precision) as clf:
            clf.classify(raw=reads.raw, offsets=reads.offsets)
            t = clf.tuning()
        route = "dealt" if t["dealt"] else {1: 1, 4: 4}.get(t["warps_per_cta"], "all")
        assert route != "all" or (t["warps_per_cta"] >= 12 and t["ctas_per_sm"] == 1)
        seen.setdefault(route, []).append(len(lengths))
    print(precision, seen)
    return set(seen)


@pytest.mark.parametrize("precision", [1, 2])
def test_default_shapes_reach_every_route(setup, precision):  # noqa: F811
    tested = params(teams.test_default_shapes_give_the_same_bits, "lengths")
    assert routes(setup, precision, tested + [MIDDLE]) == {"dealt", 1, 4, "all"}


def test_fp16_default_shapes_reach_every_route(setup):  # noqa: F811
    tested = params(teams.test_fp16_default_keeps_the_bits_of_single_warps, "n,length")
    assert routes(setup, 0, [[length] * n for n, length in tested]) == {"dealt", 1, 4, "all"}


@pytest.mark.parametrize("precision", [1, 2])
def test_teams_of_4_have_the_bits_of_single_warps(setup, precision):  # noqa: F811
    g, _, tab = setup
    reads = batch(setup, MIDDLE)
    with make_classifier(g, tab, precision=precision) as clf:
        got = clf.classify(raw=reads.raw, offsets=reads.offsets)
        assert clf.tuning()["warps_per_cta"] == 4 and not clf.tuning()["dealt"]
    with make_classifier(g, tab, precision=precision, cells_per_thread=32, chunk_strips=64, warps_per_cta=1) as clf:
        same_bits(got, clf.classify(raw=reads.raw, offsets=reads.offsets))
