"""Sweeps shared by the warps of a CTA, and the other paths a launch shape picks.

A strip's left neighbour runs on another warp, a window of rows ahead, so the
cases sit where that can go wrong: reads of one row, of a window less and more
than full, of fewer rows than the pipeline is long; more items than teams and
fewer; chunks that resume from rows their neighbours overwrite.  FP32 and MIXED
cells have the same bits for every shape, FP16 pairs for every team size at the
same chunks, REF_DEL for every shape: results are compared bit for bit with one
warp per item, and FP32 with the FP64 oracle (1e-5 relative: 2,048 rows of two
FP32 roundings, 2^-24 each, on sums of positive terms).
"""
import ctypes

import numpy as np
import pytest

from gpu_util import make_classifier, oracle_classify, small_genome
from dtwax_gb300 import synth

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 31, 32, 33, 63, 64, 65, 127, 383, 384, 385, 639, 640, 641, 799, 801, 1023, 1600, 2048]
FIELDS = ("score_fwd", "score_rev", "end_pos", "strand")


@pytest.fixture(scope="module")
def setup(built_lib):
    g, o = small_genome(26_000, 41), small_genome(26_000, 42)
    return g, o, synth.level_table()


def batch(setup, lengths, seed=6):
    g, o, tab = setup
    return synth.simulate_reads(g, o, tab, lengths, [i % 2 for i in range(len(lengths))], seed=seed)


def same_bits(a, b):
    for k in FIELDS:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("strips", [1, 5, 40])
def test_team_sizes_give_the_same_bits(setup, precision, strips):
    g, _, tab = setup
    reads = batch(setup, EDGES)
    cells = {0: 48, 1: 32, 2: 64}[precision]
    res = []
    for warps in (1, 2, 3, 4, 8):
        with make_classifier(g, tab, precision=precision, cells_per_thread=cells, chunk_strips=strips,
                             warps_per_cta=warps) as clf:
            res.append(clf.classify(raw=reads.raw, offsets=reads.offsets))
    for r in res[1:]:
        same_bits(r, res[0])


@pytest.mark.parametrize("lengths", [[2048], [300] * 70, [700] * 200, [2000] * 10, [1500] * 64, [900, 8000] * 20,
                                     EDGES * 3])
@pytest.mark.parametrize("precision", [1, 2])
def test_default_shapes_give_the_same_bits(setup, oracle, precision, lengths):
    """Dealt batches, single warps, teams of 4 and of all an SM's warps."""
    g, _, tab = setup
    reads = batch(setup, lengths)
    with make_classifier(g, tab, precision=precision) as clf:
        got = clf.classify(raw=reads.raw, offsets=reads.offsets)
    with make_classifier(g, tab, precision=precision, cells_per_thread=32, chunk_strips=64, warps_per_cta=1) as clf:
        want = clf.classify(raw=reads.raw, offsets=reads.offsets)
        same_bits(got, want)
        if precision == 1 and len(lengths) <= 60:
            sf, _, sr, _ = oracle_classify(oracle, clf, reads.raw, reads.offsets)
            np.testing.assert_allclose(got["score_fwd"], sf, rtol=1e-5, atol=1e-6)
            np.testing.assert_allclose(got["score_rev"], sr, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("n,length", [(1, 2048), (12, 2048), (40, 300), (300, 700), (30, 4000)])
def test_fp16_default_keeps_the_bits_of_single_warps(setup, n, length):
    """The default FP16 chunks, swept by the default team (dealt or not) and by
    single warps."""
    g, _, tab = setup
    reads = batch(setup, [length] * n)
    with make_classifier(g, tab, precision=0) as clf:
        got = clf.classify(raw=reads.raw, offsets=reads.offsets)
        chunk = clf.tuning()["chunk_strips"]
    with make_classifier(g, tab, precision=0, chunk_strips=chunk, warps_per_cta=1) as clf:
        same_bits(got, clf.classify(raw=reads.raw, offsets=reads.offsets))


@pytest.mark.parametrize("precision,state", [(1, 0), (2, 0), (0, 0), (0, 1)])
def test_resumed_chunks_read_rows_before_they_are_overwritten(setup, precision, state):
    """More items than the GPU has warps, one strip each: a chunk may be swept
    long after its left neighbour was.  Every read is the same read, so every
    decision has to be the one of that read alone."""
    g, _, tab = setup
    x = batch(setup, [3 * 800])
    cells, strips = (16, 1) if precision == 1 else (32, 1)
    out = []
    for reads in (1, 96):
        with make_classifier(g, tab, precision=precision, state_precision=state, threshold=-1.0,
                             cells_per_thread=cells, chunk_strips=strips) as clf:
            clf.serve_start(max_in_flight=reads, chunks_per_decision=3)
            for k in range(3):
                for r in range(reads):
                    clf.submit_chunk(r, 1 + r, x.raw[800 * k:800 * (k + 1)], is_last=k == 2)
                clf.serve_step()
                clf.serve_drain()
            out.append({(d["read_number"], d["chunks"]): (d["score"], d["end_pos"], d["strand"])
                        for d in clf.poll_decisions(4096)})
    assert len(out[0]) == 3 and len(out[1]) == 3 * 96
    for (_, chunks), d in out[1].items():
        assert d == out[0][(1, chunks)]


@pytest.mark.parametrize("precision,cells", [(1, 16), (1, 32), (0, 32)])
@pytest.mark.parametrize("lengths", [EDGES, [1999, 2000] * 40, [96] * 700, [1500] * 3])
def test_ref_del_teams_give_the_same_bits(built_lib, precision, cells, lengths):
    """Teams of every default size against one warp per read (odd row counts
    end on a lane's first row)."""
    import dtwax_gb300 as d
    g, o = small_genome(70_000, 43), small_genome(70_000, 44)
    tab = synth.level_table()
    reads = synth.simulate_reads(g, o, tab, lengths, [i % 2 for i in range(len(lengths))], seed=3)
    res = []
    for warps in (0, 1):
        with make_classifier(g, tab, precision=precision, recurrence=d.REF_DEL, cells_per_thread=cells,
                             warps_per_cta=warps) as clf:
            res.append(clf.classify(raw=reads.raw, offsets=reads.offsets))
    same_bits(res[0], res[1])


@pytest.mark.parametrize("m", [507, 512, 1500, 1537, 6000])
@pytest.mark.parametrize("lengths", [[1], [33, 2048], [700] * 90, [2048] * 30])
def test_static_entry_has_the_bits_of_the_regular_one(built_lib, m, lengths):
    """Reference lengths around the 512-column padding and the strip width; the
    padding is the last thing in its allocation."""
    import torch
    import dtwax_gb300 as d
    lib = d.load_library()
    g, o = small_genome(m + 5, 45), small_genome(m + 5, 46)
    tab = synth.level_table()
    reads = synth.simulate_reads(g, o, tab, lengths, [i % 2 for i in range(len(lengths))], seed=2)
    n = reads.n
    with make_classifier(g, tab, precision=1) as clf:
        fwd, rev = clf.reference()
        raw = torch.tensor(reads.raw, device="cuda")
        q = torch.zeros_like(raw)
        clf.normalize(raw.data_ptr(), reads.offsets, q.data_ptr())
        pairs = torch.zeros((-(-m // 512) * 512, 2), device="cuda")
        pairs[:m] = torch.tensor(np.stack([fwd, rev], 1), device="cuda")
        outs = [torch.zeros(32 * n, dtype=torch.uint8, device="cuda") for _ in range(2)]
        clf.distances(q.data_ptr(), reads.offsets, outs[0].data_ptr())
        rc = lib.dtwx_distances_static(ctypes.c_void_p(pairs.data_ptr()), m, ctypes.c_void_p(q.data_ptr()),
                                       reads.offsets.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)), n,
                                       ctypes.c_float(clf.cfg.threshold), ctypes.c_void_p(outs[1].data_ptr()), None)
        assert rc == 0
        torch.cuda.synchronize()
    a, b = (np.frombuffer(t.cpu().numpy().tobytes(), d.RESULT_DTYPE) for t in outs)
    same_bits(a, b)


@pytest.mark.parametrize("kind", ["pA", "offset", "counts", "constant", "huge", "tiny", "nan"])
def test_normalizer_rounds_the_64_bit_value(built_lib, kind):
    """Lengths around a block and the staging limit, and inputs on both sides of
    the float-pair path's range.  The result is the FP64 value rounded to FP32
    up to one unit in the last place (numpy's own sums differ from any other
    order in their last bits)."""
    import torch
    rng = np.random.default_rng(9)
    lens = np.array([1, 2, 31, 255, 256, 257, 4999, 11_776, 11_777, 30_000])
    offsets = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    x = rng.standard_normal(int(offsets[-1]))
    x = {"pA": 90 + 12 * x, "offset": 1e6 + x, "counts": np.round(400 + 60 * x), "constant": 0 * x + 90.25,
         "huge": 1e18 * x, "tiny": 1e-15 * x, "nan": np.where(np.arange(x.size) == 40, np.nan, x)}[kind]
    x = x.astype(np.float32)
    for eps in (1e-4, 0.0) if kind != "constant" else (1e-4,):
        with make_classifier(small_genome(3000), precision=1, norm_eps=eps) as clf:
            raw = torch.tensor(x, device="cuda")
            y = torch.zeros_like(raw)
            clf.normalize(raw.data_ptr(), offsets, y.data_ptr())
            y = y.cpu().numpy()
        for r in range(1 if eps == 0.0 else 0, lens.size):  # (one sample has no spread)
            v = x[offsets[r]:offsets[r + 1]].astype(np.float64)
            want = ((v - v.mean()) / np.sqrt(((v - v.mean()) ** 2).mean() + np.float64(np.float32(eps)))).astype(np.float32)
            np.testing.assert_array_max_ulp(y[offsets[r]:offsets[r + 1]], want, maxulp=1) \
                if not np.isnan(want).any() else np.testing.assert_array_equal(np.isnan(y[offsets[r]:offsets[r + 1]]), np.isnan(want))


@pytest.mark.parametrize("length,cap,concat", [(6, 0, 0), (4101, 0, 0), (4102, 0, 1), (9000, 3000, 0), (9000, 4097, 1)])
def test_reference_builder_at_its_edges(built_lib, oracle, length, cap, concat):
    """Genomes around a CTA's 4,096 columns, a capped one, invalid bases at both
    ends and in the middle."""
    g = bytearray(small_genome(length, 47))
    if length > 100:
        for i in (0, length // 2, length - 1):
            g[i] = ord("N")
    g = bytes(g)
    tab = synth.level_table()
    with make_classifier(g, tab, precision=1, max_ref_len=cap, strand_mode=concat) as clf:
        fwd, rev = clf.reference()
    with np.errstate(invalid="ignore"):
        of, orv = oracle.build_levels(g, np.asarray(tab, np.float64), cap=cap)
    # levels without spread (one k-mer): 0 / 0 in the oracle, 0 in the library
    np.testing.assert_allclose(fwd, np.nan_to_num(of), atol=2e-6)
    np.testing.assert_allclose(rev, np.nan_to_num(orv), atol=2e-6)
