"""Phase B by regions. On the host, what lets a region run in one CTA and every
wait end (tests/cpp/regions.cu). On the GPU, the same frames decoded by regions
and by chains (a traced frame runs by chains), which must give the same
samples: regions cut by the picture's sides, regions of one block, blocks of
several items, raw residuals, each bit depth and superblock size; and layouts
and coding orders that no partition tree gives (tests/cpp/layouts.hpp), in
4:2:0, 4:2:2 and 4:4:4."""
import os
import subprocess

import numpy as np
import pytest

import test_plan_invariants as tpi
from test_plan_invariants import have_nvcc  # noqa: F401


def _run_checker(tmp_path, name, opt='-O2'):
    from av1ongpu_b200 import build as b
    b.build()
    objs = [os.path.join(b.OUT, f) for f in ('kernels.cu.o', 'plan_host.cpp.o', 'synth.cpp.o', 'blob.cpp.o',
                                             'api.cpp.o', 'noalloc.cu.o')]
    exe = str(tmp_path / name)
    cmd = [tpi.NVCC, '-gencode', 'arch=compute_100a,code=sm_100a', opt, '-std=c++17', '-diag-suppress', '68',
           '-I', tpi.CSRC, '-I', os.path.join(tpi.ROOT, 'include'),
           os.path.join(tpi.ROOT, 'tests', 'cpp', name + '.cu')] + objs + ['-o', exe, '-lpthread']
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    assert r.stdout.strip().endswith('ok')


def test_regions_only_wait_on_earlier_items(tmp_path, have_nvcc):  # noqa: F811
    _run_checker(tmp_path, 'regions')


def test_regions_cost_a_small_part_of_the_plan(tmp_path, have_nvcc):  # noqa: F811
    _run_checker(tmp_path, 'plan_cost', '-O3')


def _decode(av1b, params, frames, traced):
    d = av1b.Decoder(0)
    d.set_unit_trace(traced)
    slots, out = [], []
    for k in range(frames):
        b = av1b.synth_frame_ex(*params[:6], 97, k, params[6])
        b.set_refs([slots[k - x] for x in b.get_refs()])
        slot, planes = d.decode(b)
        slots.append(slot)
        out.append(planes)
    d.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize('params', [
    (16, 16, 0, 8, 64, 'all', 30),
    (64, 64, 0, 10, 64, 'all', 30),
    (66, 130, 0, 8, 64, 'all', 30),
    (150, 90, 112, 12, 128, 'all', 30),
    (240, 136, 0, 10, 64, 'residual', 30),
    (998, 514, 750, 12, 128, 'all', 2),
    (1366, 766, 0, 8, 128, 'all', 30),
    (1920, 1080, 0, 10, 64, 'all', 30),
])
def test_regions_and_chains_agree(av1b, params):
    if not av1b.cuda_available():
        pytest.skip('no CUDA device')
    tools = {'all': av1b.TOOLS_ALL, 'residual': av1b.TOOLS_ALL | av1b.TOOL_RESIDUAL}
    prm = params[:5] + (tools[params[5]],) + params[6:]
    for k, (a, b) in enumerate(zip(_decode(av1b, prm, 3, False), _decode(av1b, prm, 3, True))):
        for p in range(3):
            assert np.array_equal(a[p], b[p]), 'frame %d plane %d' % (k, p)


def build_layouts_client(tmp_path):
    exe = str(tmp_path / 'layouts_client')
    lib = os.path.join(tpi.ROOT, 'av1ongpu_b200')
    cmd = ['/usr/bin/g++', '-std=c++17', '-O1', os.path.join(tpi.ROOT, 'tests', 'cpp', 'layouts_client.cpp'),
           '-L', lib, '-lav1b', '-Wl,-rpath,' + lib, '-o', exe]
    subprocess.run(cmd, check=True, capture_output=True)
    return exe


def test_layouts_client_builds(tmp_path):
    from av1ongpu_b200 import build as b
    b.build()
    build_layouts_client(tmp_path)


@pytest.mark.gpu
def test_layouts_by_regions_and_by_chains(av1b, tmp_path):
    if not av1b.cuda_available():
        pytest.skip('no CUDA device')
    r = subprocess.run([build_layouts_client(tmp_path)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith('ok'), r.stdout[-2000:] + r.stderr[-500:]
