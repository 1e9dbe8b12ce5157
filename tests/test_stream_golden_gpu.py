"""The device-resident stream against the committed hashes of the oracle's
output (tests/golden/oracle_hashes.json): every shown reconstruction of the
small golden clips, in output order. The clips cover the turbo tool set, every
tool on an odd-sized picture (transform type and depth search, compound,
loop restoration), the low-delay path with forced loop-restoration units, and
lossless coding; no oracle build is needed. Loop-restoration units at the
sizes where the search's layout changes are checked against the oracle where
it is built."""
import hashlib
import json
import os

import numpy as np
import pytest

import mav1cu
import oracle
import parity
import synthetic

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
GOLDEN = json.load(open(os.path.join(HERE, "golden", "oracle_hashes.json")))
# clip and flags of each golden entry (tests/golden/make_golden.py)
CASES = {
    "c0_turbo_q125": (dict(width=352, height=288, frames=30, seed=1), dict(q=125, turbo=1, keyint=30, tiles=0)),
    "full_203x131": (dict(width=203, height=131, frames=9, seed=41, rects=3, rect_size=(16, 48)),
                     dict(q=90, altref=4, golden=1, tiles=1, me_range=64)),
    "lowdelay_lr_150x102": (dict(width=150, height=102, frames=6, seed=42, rects=2, rect_size=(16, 40)),
                            dict(q=200, golden=1, keyint=4, lr_test=1)),
    "lossless_96x64": (dict(width=96, height=64, frames=3, seed=43, rects=1, rect_size=(16, 32)), dict(q=0, fast=1)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_stream_reconstructions_match_golden(name):
    import torch
    kw, flags = CASES[name]
    spec = synthetic.ClipSpec(**kw)
    assert synthetic.clip_sha256(spec) == GOLDEN[name]["clip"]
    clip = [torch.from_numpy(np.frombuffer(synthetic.packed(f), np.uint8).copy()).cuda() for f in synthetic.generate(spec)]
    torch.cuda.synchronize()
    cfg = mav1cu.cli_config(spec.width, spec.height, **flags)
    g = mav1cu.geometry(spec.width, spec.height)
    st = mav1cu.Stream(cfg)
    shown, slots = [], [None] * 8
    try:
        for job in mav1cu.plan(cfg, spec.frames):
            sess = st.encode(job, clip[int(job["disp"])].data_ptr(), True)
            st.synchronize()
            rec = parity.visible(sess.download("REC", count=g["frame_bytes"]), g)
            sha = hashlib.sha256(rec.tobytes()).hexdigest()[:16]
            for k in range(8):
                if (0xFF if job["is_key"] else int(job["refresh"])) >> k & 1:
                    slots[k] = sha
            if not job["hidden"]:
                shown.append(sha)
            if job["show_existing"] >= 0:
                shown.append(slots[int(job["show_existing"])])
    finally:
        st.close()
    assert shown == GOLDEN[name]["recon_sha16"]


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
