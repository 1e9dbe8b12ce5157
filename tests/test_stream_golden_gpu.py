"""The device-resident stream against committed hashes; no oracle build is
needed. Every shown reconstruction of the small golden clips, in output order,
against the oracle's (golden/oracle_hashes.json): the turbo tool set, every
tool on an odd-sized picture (transform type and depth search, compound, loop
restoration), the low-delay path with forced loop-restoration units, and
lossless coding. And every exported image of the clips of parity.stream_clips
against golden/stream_hashes.json, and the restoration units of made-up frames
against golden/lr_hashes.json (golden/make_golden.py --stream says where they
come from): picture sizes at the edges of the kernels' tiles, restoration
units at the sizes where the search's layout changes, and more units than a
round of its choice takes. Where the oracle is built, the same clips are
compared with it, stage by stage."""
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
HASHES = json.load(open(os.path.join(HERE, "golden", "stream_hashes.json")))
LR_HASHES = json.load(open(os.path.join(HERE, "golden", "lr_hashes.json")))


@pytest.mark.parametrize("name", sorted(parity.GOLDEN_CLIPS))
def test_stream_reconstructions_match_golden(name):
    shown, want = parity.golden_stream(name)
    assert shown == want


@pytest.mark.parametrize("name", sorted(parity.stream_clips()))
def test_stream_images_match_golden(name):
    spec, flags = parity.stream_clips()[name]
    assert synthetic.clip_sha256(spec) == HASHES[name]["clip"]
    assert [parity.sha16(i) for i in parity.stream_images(spec, flags)] == HASHES[name]["image_sha16"]


@pytest.mark.parametrize("w,h", parity.LR_FRAMES)
def test_lr_units_match_golden(w, h):
    want = LR_HASHES[f"{w}x{h}"]
    assert parity.sha16(np.concatenate(parity.lr_frame(w, h, 3 * w + h))) == want["frame"]
    for lr_test in (0, 1):
        units, types = parity.lr_units(w, h, lr_test)
        assert parity.sha16(units) + parity.sha16(types) == want["units"][lr_test]
        assert np.bincount(units["type"], minlength=3).tolist() == want["types"][lr_test]
    # the frames are worth searching: the large ones keep all three kinds of unit
    assert w * h < 200000 or min(want["types"][0]) > 0


# the least room (every round overflows, the caches refill), little, and a round of one warp a unit
@pytest.mark.parametrize("lr_test", [0, 1])
@pytest.mark.parametrize("room", [(1, 25), (5, 26), (8, 40)])
def test_lr_choice_does_not_depend_on_its_room(room, lr_test):
    units, types = parity.lr_units(640, 360, lr_test, room=room)
    assert parity.sha16(units) + parity.sha16(types) == LR_HASHES["640x360"]["units"][lr_test]


def test_lr_search_refuses_units_its_windows_cannot_hold():
    s = mav1cu.Session(159, 159)
    try:
        assert s.lib.mav1cu_debug_lr_room(s.h, 0, 40) == -1
    finally:
        s.close()
    s = mav1cu.Session(159, 159)
    try:
        cfg = mav1cu.cli_config(159, 159, q=100)
        fp, _ = mav1cu.frame_params(cfg, mav1cu.plan(cfg, 1)[0])
        p = fp.view(mav1cu.PARAMS_DTYPE)
        p["lr_unit_size"], p["lr_unit_rows"], p["lr_unit_cols"], p["lr_unit_off"] = 128, 1, 1, [0, 1, 2]
        s.set_params(fp)
        assert s.lib.mav1cu_lr_search(s.h, 0) == -1
    finally:
        s.close()


@pytest.mark.skipif(not oracle.available(), reason="oracle not built")
@pytest.mark.parametrize("w,h", parity.LR_SIZES)
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


@pytest.mark.skipif(not oracle.available(), reason="oracle not built")
@pytest.mark.parametrize("tools", sorted(parity.STREAM_TOOLS))
@pytest.mark.parametrize("w,h", parity.STREAM_SIZES)
def test_stream_sizes_match_oracle(w, h, tools):
    spec = synthetic.ClipSpec(w, h, 4, seed=w + 3 * h, rects=3, rect_size=(8, 32))
    tr, _, frames, _, _ = parity.trace_clip(spec, 4, **parity.STREAM_TOOLS[tools])
    bad = [(k, o) for k, o in parity.stream_vs_oracle(tr, frames, parity.STREAM_TOOLS[tools], spec) if any(o.values())]
    assert not bad, bad
