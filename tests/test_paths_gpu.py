"""The kernels' size and type rules at the places where a path begins or ends:
superres by 1:2 (the widest prediction window) to 8:9, sides that are no
multiple of a tile, one tile, 12-bit samples (wider sums), streams without
restoration, grain, deblocking or CDEF (other picture buffers), lossless
blocks, and frames large enough for the launches that small ones merge.
Every frame's planes and NV12 pack against hashes the decoder gave before
these paths existed, when it matched the reference's CPU backend on every
parity test (tests/golden/paths.json), and against that backend itself where
it is built."""
import hashlib
import json
import os

import numpy as np
import pytest

PATHS = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'golden', 'paths.json')


def cases(A):
    ext = A.TOOLS_ALL | A.TOOL_INTERINTRA | A.TOOL_INTRABC | A.TOOL_RESIDUAL
    plain = A.TOOLS_ALL & ~(A.TOOL_LR | A.TOOL_GRAIN)
    # name: (width, height, coded_width, bit_depth, superblock, tools, key_interval), frames
    return {
        'superres_half': ((256, 144, 128, 10, 64, A.TOOLS_ALL, 30), 4),
        'superres_half_odd': ((198, 134, 99, 8, 128, ext, 30), 4),
        'superres_8_9': ((360, 200, 320, 12, 64, A.TOOLS_ALL, 30), 3),
        'superres_no_lr': ((320, 182, 200, 10, 64, plain, 30), 3),
        'sides_off_tiles': ((338, 206, 0, 8, 64, ext, 30), 4),
        'one_tile': ((16, 16, 0, 10, 64, A.TOOLS_ALL, 30), 3),
        'twelve_bits': ((330, 186, 0, 12, 128, ext, 30), 3),
        'no_filters': ((200, 120, 0, 10, 64, plain | A.TOOL_NO_DEBLOCK | A.TOOL_NO_CDEF, 30), 4),
        'restoration_only': ((200, 120, 0, 10, 64, (A.TOOLS_ALL & ~A.TOOL_GRAIN) | A.TOOL_NO_DEBLOCK |
                              A.TOOL_NO_CDEF, 30), 4),
        'cdef_only': ((264, 152, 0, 8, 64, plain | A.TOOL_NO_DEBLOCK, 30), 3),
        'lossless': ((168, 104, 0, 8, 64, A.TOOL_LOSSLESS, 0), 2),
        'larger': ((1416, 798, 0, 10, 64, A.TOOLS_ALL, 30), 3),
        'larger_masks': ((1922, 1082, 0, 8, 128, ext, 30), 3),
    }


def frames(dec, av1b, params, n, keep):
    """Hashes of each frame's planes and of its NV12 pack. keep: every frame
    into a slot; else the last one is decoded without."""
    w, h = params[:2]
    pitch = (w + 63) & ~63
    slots, out = [], []
    for k in range(n):
        b = av1b.synth_frame_ex(*params[:6], 808, k, params[6])
        b.set_refs([slots[k - x] for x in b.get_refs()])
        slot, planes = dec.decode(b, keep=keep or k < n - 1)
        slots.append(slot)
        hsh = hashlib.sha256()
        for p in planes:
            hsh.update(np.ascontiguousarray(p).tobytes())
        hsh.update(dec.to_nv12(slot, pitch, w, h).tobytes())
        out.append(hsh.hexdigest()[:32])
    for s in slots:
        if s >= 0:
            dec.release_reference(s)
    return out


NAMES = ['superres_half', 'superres_half_odd', 'superres_8_9', 'superres_no_lr', 'sides_off_tiles', 'one_tile',
         'twelve_bits', 'no_filters', 'restoration_only', 'cdef_only', 'lossless', 'larger', 'larger_masks']


@pytest.mark.gpu
@pytest.mark.parametrize('keep', [True, False])
@pytest.mark.parametrize('name', NAMES)
def test_frames_of_a_path(av1b, name, keep):
    if not av1b.cuda_available():
        pytest.skip('no CUDA device')
    params, n = cases(av1b)[name]
    dec = av1b.Decoder(0)
    got = frames(dec, av1b, params, n, keep)
    dec.close()
    assert got == json.load(open(PATHS))[name]


@pytest.mark.gpu
@pytest.mark.parametrize('name', NAMES)
def test_planned_frames_of_a_path(av1b, name):
    """The same frames planned ahead and queued, each packed on the device: the
    pack that applies the grain, and no wait between frames."""
    import torch
    if not av1b.cuda_available():
        pytest.skip('no CUDA device')
    params, n = cases(av1b)[name]
    w, h = params[:2]
    pitch = (w + 63) & ~63
    dec = av1b.Decoder(0)
    slots = [dec.reserve_reference() for _ in range(n)]
    size = av1b.nv12_size(w, h, 1, 1, pitch)
    bufs = [torch.zeros(size, dtype=torch.uint8, device='cuda') for _ in range(n)]
    torch.cuda.synchronize()
    plans, want = [], []
    for k in range(n):
        b = av1b.synth_frame_ex(*params[:6], 808, k, params[6])
        b.set_refs([slots[k - x] for x in b.get_refs()])
        plans.append(dec.plan(b))
    for k in range(n):
        dec.decode_planned(plans[k], slot=slots[k], wait=False)
        dec.to_nv12_device(slots[k], pitch, bufs[k].data_ptr(), size)
    dec.sync()
    for k in range(n):
        planes = [np.empty(s, dtype=np.uint16) for s in av1b.plane_shapes(w, h, 1, 1)]
        dec.decode_planned(plans[k], slot=slots[k], wait=True, planes=planes)
        hsh = hashlib.sha256()
        for p in planes:
            hsh.update(p.tobytes())
        hsh.update(bufs[k].cpu().numpy().tobytes())
        want.append(hsh.hexdigest()[:32])
    for p in plans:
        dec.free_plan(p)
    dec.close()
    assert want == json.load(open(PATHS))[name]


@pytest.mark.gpu
@pytest.mark.parametrize('name', NAMES)
def test_frames_of_a_path_against_the_reference(av1b, oracle, name):
    params, n = cases(av1b)[name]
    assert frames(oracle.RefDecoder(), av1b, params, n, True) == json.load(open(PATHS))[name]


def test_packed_filter_ranges():
    """What the packed prediction relies on: every subpel tap is even with a
    half that fits 8 bits, and the intermediate of a 12-bit picture (the sum
    rounded by five bits; three for 10 bits) fits 16."""
    import re
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    text = open(os.path.join(root, 'av1ongpu_b200', 'csrc', 'av1b_tables.h')).read()
    taps = [int(v) for v in re.findall(r'-?\d+', re.search(r'kSubpelFilters\[768\] = \{(.*?)\}', text, re.S).group(1))]
    assert len(taps) == 768
    assert all(v % 2 == 0 and -128 <= v // 2 <= 127 for v in taps)
    rows = [taps[i:i + 8] for i in range(0, 768, 8)]
    for top, shift in ((4095, 5), (1023, 3), (255, 3)):
        assert max(sum(v for v in r if v > 0) for r in rows) * top >> shift < 32768
        assert min(sum(v for v in r if v < 0) for r in rows) * top >> shift >= -32768
    # the window loop's k / n by a multiply and a shift
    recip = [(65536 + n - 1) // n for n in range(1, 13)]
    src = open(os.path.join(root, 'av1ongpu_b200', 'csrc', 'dev_inter.cuh')).read()
    table = [int(v) for v in re.findall(r'\d+', re.search(r'kRecip16\[13\] = \{(.*?)\}', src, re.S).group(1))]
    assert table == [0] + recip
    assert all(k * r >> 16 == k // (n + 1) for n, r in enumerate(recip) for k in range(15 * 12))
