"""Phase B's waits on tagged samples. On the host, the planner's cell masks
against the dependency lists they stand for (tests/cpp/wait_cells.cu). On the
GPU, the same frames decoded with tags and with done flags (a traced frame
waits on done flags only), which must give the same samples, and a decoder
that has used up its 65,535 tags and starts over."""
import os
import subprocess

import numpy as np
import pytest

import test_plan_invariants as tpi
from test_plan_invariants import have_nvcc  # noqa: F401


def test_cell_masks_are_the_dependency_lists(tmp_path, have_nvcc):  # noqa: F811
    from av1ongpu_b200 import build as b
    b.build()
    objs = [os.path.join(b.OUT, f) for f in ('kernels.cu.o', 'plan_host.cpp.o', 'synth.cpp.o', 'blob.cpp.o',
                                             'api.cpp.o', 'noalloc.cu.o')]
    exe = str(tmp_path / 'wait_cells')
    cmd = [tpi.NVCC, '-gencode', 'arch=compute_100a,code=sm_100a', '-O2', '-std=c++17', '-diag-suppress', '68',
           '-I', tpi.CSRC, '-I', os.path.join(tpi.ROOT, 'include'),
           os.path.join(tpi.ROOT, 'tests', 'cpp', 'wait_cells.cu')] + objs + ['-o', exe, '-lpthread']
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    assert r.stdout.strip().endswith('ok')


def _decode(av1b, params, frames, traced):
    d = av1b.Decoder(0)
    d.set_unit_trace(traced)
    slots, out = [], []
    for k in range(frames):
        b = av1b.synth_frame_ex(*params[:6], 321, k, params[6])
        b.set_refs([slots[k - x] for x in b.get_refs()])
        slot, planes = d.decode(b)
        slots.append(slot)
        out.append(planes)
    d.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize('params', [
    (16, 16, 0, 8, 64, 'all', 30),
    (150, 90, 0, 8, 64, 'all', 2),
    (150, 90, 112, 12, 128, 'all', 30),
    (240, 136, 0, 10, 64, 'extended', 30),
    (1366, 766, 0, 8, 128, 'extended', 30),
    (1280, 720, 0, 8, 64, 'basic', 0),
])
def test_tags_and_flags_agree(av1b, params):
    if not av1b.cuda_available():
        pytest.skip('no CUDA device')
    tools = {'basic': 0, 'all': av1b.TOOLS_ALL,
             'extended': av1b.TOOLS_ALL | av1b.TOOL_INTERINTRA | av1b.TOOL_INTRABC | av1b.TOOL_RESIDUAL}
    prm = params[:5] + (tools[params[5]],) + params[6:]
    for k, (a, b) in enumerate(zip(_decode(av1b, prm, 3, False), _decode(av1b, prm, 3, True))):
        for p in range(3):
            assert np.array_equal(a[p], b[p]), 'frame %d plane %d' % (k, p)


@pytest.mark.gpu
def test_tags_start_over(av1b):
    if not av1b.cuda_available():
        pytest.skip('no CUDA device')
    d = av1b.Decoder(0)
    b = av1b.synth_frame_ex(16, 16, 0, 8, 64, 0, 9, 0, 0)
    _, want = d.decode(b, keep=False)
    plan = d.plan(b)
    for k in range(65600):
        d.decode_planned(plan, keep=False, wait=k % 512 == 0)
    d.sync()
    planes = [np.empty(a.shape, dtype=np.uint16) for a in want]
    d.decode_planned(plan, keep=False, wait=True, planes=planes)
    d.free_plan(plan)
    d.close()
    for p in range(3):
        assert np.array_equal(planes[p], want[p])
