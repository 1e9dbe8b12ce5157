"""The device-resident stream against the committed hashes of the oracle's
output (tests/golden/oracle_hashes.json): every shown reconstruction of the
small golden clips, in output order. The clips cover the turbo tool set, every
tool on an odd-sized picture (transform type and depth search, compound,
loop restoration), the low-delay path with forced loop-restoration units, and
lossless coding; no oracle build is needed. Loop-restoration units at the
sizes where the search's layout changes are checked against the oracle where
it is built."""
import pytest

import mav1cu
import oracle
import parity
import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", sorted(parity.GOLDEN_CLIPS))
def test_stream_reconstructions_match_golden(name):
    shown, want = parity.golden_stream(name)
    assert shown == want


# one unit narrower and lower than 64 samples, the largest units (95 columns, 103 luma / 99 chroma rows), units
# cut mid-stripe, several units a row with a remainder of one block
@pytest.mark.skipif(not oracle.available(), reason="oracle not built")
@pytest.mark.parametrize("w,h", [(48, 40), (95, 95), (159, 159), (191, 190), (130, 98), (67, 223)])
def test_lr_search_unit_sizes(w, h):
    spec = synthetic.ClipSpec(w, h, 2, seed=w * 7 + h, rects=2, rect_size=(12, 30))
    tr, cfg, _, _, _ = parity.trace_clip(spec, 2, q=120, golden=1, tiles=0)
    sess = mav1cu.Session(w, h)
    try:
        bad = [(k, out) for k, fr in enumerate(tr.frames) for out in [parity.FrameCheck(sess, tr, cfg, fr).lr_search()]
               if any(out.values())]
    finally:
        sess.close()
    assert not bad, bad


# pictures of one superblock and of less, of partial superblocks on either side, of several tile columns, a wide
# one of one superblock row: the edges of the dataflow's records, the filter tiles and the refinement windows
SIZES = [(64, 64), (72, 72), (130, 66), (66, 194), (392, 40), (264, 136)]
TOOLS = {
    "turbo": dict(q=110, turbo=1, keyint=4, tiles=1),
    "full": dict(q=90, altref=4, golden=1, tiles=1, me_range=64),
    "lossless": dict(q=0, fast=1),
}


@pytest.mark.skipif(not oracle.available(), reason="oracle not built")
@pytest.mark.parametrize("tools", sorted(TOOLS))
@pytest.mark.parametrize("w,h", SIZES)
def test_stream_sizes_match_oracle(w, h, tools):
    spec = synthetic.ClipSpec(w, h, 4, seed=w + 3 * h, rects=3, rect_size=(8, 32))
    tr, _, frames, _, _ = parity.trace_clip(spec, 4, **TOOLS[tools])
    bad = [(k, o) for k, o in parity.stream_vs_oracle(tr, frames, TOOLS[tools], spec) if any(o.values())]
    assert not bad, bad
