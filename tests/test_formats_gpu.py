"""Chroma formats and frames without some stages: 4:2:2 and 4:4:4 frames of
every tool (the regions' tiles, tiled CDEF's cells, the packed prediction's
windows and the grain templates in those formats), film grain in frames that
nothing else filters, and inter frames without a block of the dependency-
scheduled phase. Every frame's planes against hashes the decoder gave before
those paths existed, when it matched the reference's CPU backend on streams of
each format (tests/golden/formats.json), and against that backend itself where
it is built."""
import hashlib
import json
import os

import numpy as np
import pytest

FORMATS = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'golden', 'formats.json')


def cases(A):
    ext = A.TOOLS_ALL | A.TOOL_INTERINTRA | A.TOOL_INTRABC | A.TOOL_RESIDUAL
    # name: (width, height, coded_width, bit_depth, superblock, tools), frames
    return {
        '422': ((338, 206, 0, 8, 64, ext | A.TOOL_422), 3),
        '444': ((338, 206, 0, 10, 64, ext | A.TOOL_444), 3),
        '422_superres': ((360, 200, 270, 12, 128, A.TOOLS_ALL | A.TOOL_422), 3),
        '444_superres': ((320, 182, 200, 8, 128, A.TOOLS_ALL | A.TOOL_444), 3),
        '422_larger': ((1416, 798, 0, 10, 128, A.TOOLS_ALL | A.TOOL_422), 2),
        '444_larger': ((1416, 798, 0, 8, 64, A.TOOLS_ALL | A.TOOL_444), 2),
        'grain_alone': ((200, 120, 0, 10, 64,
                         (A.TOOLS_ALL & ~A.TOOL_LR) | A.TOOL_NO_DEBLOCK | A.TOOL_NO_CDEF), 4),
        'few_blocks': ((32, 24, 0, 8, 64, A.TOOLS_ALL), 12),
        'few_blocks_unfiltered': ((40, 24, 0, 10, 64,
                                   (A.TOOLS_ALL & ~A.TOOL_LR) | A.TOOL_NO_DEBLOCK | A.TOOL_NO_CDEF), 12),
    }


NAMES = ['422', '444', '422_superres', '444_superres', '422_larger', '444_larger', 'grain_alone', 'few_blocks',
         'few_blocks_unfiltered']


def frames(dec, av1b, params, n):
    """Hashes of each frame's planes."""
    slots, out = [], []
    for k in range(n):
        b = av1b.synth_frame_ex(*params, 515, k, 30)
        b.set_refs([slots[k - x] for x in b.get_refs()])
        slot, planes = dec.decode(b)
        slots.append(slot)
        hsh = hashlib.sha256()
        for p in planes:
            hsh.update(np.ascontiguousarray(p).tobytes())
        out.append(hsh.hexdigest()[:32])
        if len(slots) > 3:
            dec.release_reference(slots[-4])
    return out


@pytest.mark.gpu
@pytest.mark.parametrize('name', NAMES)
def test_frames_of_a_format(av1b, name):
    if not av1b.cuda_available():
        pytest.skip('no CUDA device')
    params, n = cases(av1b)[name]
    dec = av1b.Decoder(0)
    got = frames(dec, av1b, params, n)
    dec.close()
    assert got == json.load(open(FORMATS))[name]


@pytest.mark.gpu
@pytest.mark.parametrize('name', NAMES)
def test_planned_frames_of_a_format(av1b, name):
    """The same frames planned ahead and queued without a wait between them;
    the inter frames of few blocks include some without the dependency-
    scheduled phase."""
    if not av1b.cuda_available():
        pytest.skip('no CUDA device')
    params, n = cases(av1b)[name]
    w, h, tools = params[0], params[1], params[5]
    ss_x, ss_y = int(not tools & av1b.TOOL_444), int(not tools & (av1b.TOOL_422 | av1b.TOOL_444))
    dec = av1b.Decoder(0)
    slots = [dec.reserve_reference() for _ in range(4)]
    plans, none = [], 0
    # enough plans ahead that a frame is queued while the one before it runs
    for k in range(n):
        b = av1b.synth_frame_ex(*params, 515, k, 30)
        b.set_refs([slots[(k - x) % 4] for x in b.get_refs()])
        plans.append(dec.plan(b))
        none += k > 0 and dec.plan_stats(plans[-1])['phase_b_blocks'] == 0
    if name.startswith('few_blocks'):
        assert none > 0
    want = json.load(open(FORMATS))[name]
    # the planes of the last frame, then of the last but one, ..: every frame's
    # grain and filters behind the ones of the frames queued before it
    for last in range(n - 1, max(-1, n - 5), -1):
        for k in range(last):
            dec.decode_planned(plans[k], slot=slots[k % 4], wait=False)
        planes = [np.empty(s, dtype=np.uint16) for s in av1b.plane_shapes(w, h, ss_x, ss_y)]
        dec.decode_planned(plans[last], slot=slots[last % 4], wait=True, planes=planes)
        hsh = hashlib.sha256()
        for p in planes:
            hsh.update(p.tobytes())
        assert hsh.hexdigest()[:32] == want[last], last
    for p in plans:
        dec.free_plan(p)
    dec.close()


@pytest.mark.gpu
@pytest.mark.parametrize('name', NAMES)
def test_frames_of_a_format_against_the_reference(av1b, oracle, name):
    params, n = cases(av1b)[name]
    assert frames(oracle.RefDecoder(), av1b, params, n) == json.load(open(FORMATS))[name]
