"""Kernels that are launched before the ones ahead of them in the stream have
ended (launch_chained): each waits for those on every path before it ends, and
reads nothing that a kernel of the frame writes as read-only data, whose loads
may be moved above the wait. Shown from the source: a run that comes out right
shows one build on one GPU only."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'av1ongpu_b200', 'csrc')

# what the planner uploaded or wrote before the frame's first kernel
PLANNED = {'cells', 'pos', 'recs', 'coef', 'orbit'}


def _text():
    src = open(os.path.join(CSRC, 'kernels.cu')).read()
    return re.sub(r'/\*.*?\*/|//[^\n]*', '', src, flags=re.S)


def _function(src, name):
    """(parameters, body) of a function's definition."""
    for m in re.finditer(r'\b%s\(' % name, src):
        i, depth = m.end(), 1
        while depth:
            depth += {'(': 1, ')': -1}.get(src[i], 0)
            i += 1
        params, rest = src[m.end():i - 1], src[i:]
        if not rest.lstrip().startswith('{'):
            continue
        start = i + rest.index('{')
        i, depth = start + 1, 1
        while depth:
            depth += {'{': 1, '}': -1}.get(src[i], 0)
            i += 1
        return params, src[start:i]
    raise AssertionError('no definition of ' + name)


def _early_kernels(src):
    names = set(re.findall(r'launch_chained\([^,;]*,\s*(k_\w+)', src))
    assert names >= {'k_itx', 'k_inter_simple', 'k_deblock', 'k_cdef_search', 'k_cdef_tile',
                     'k_upscale', 'k_lr_tile'}
    return sorted(names)


def test_early_kernels_wait():
    src = _text()
    for name in _early_kernels(src):
        body = _function(src, name)[1]
        wait = 'ends_after_deps();' if 'ends_after_deps();' in body else 'deps_done();'
        assert body.count(wait) == 1, name
        before, after = body.split(wait)
        assert 'return' not in before, name + ' may end before it waits'
        # not inside a branch
        assert before.count('{') - before.count('}') == 1, name
        if wait == 'ends_after_deps();':
            assert after.strip() == '}', name
    # the CTA that waits for the grid is one that every grid has
    assert _function(src, 'ends_after_deps')[1].split() == \
        '{ if (blockIdx.x == gridDim.x - 1) deps_done(); }'.split()


def test_early_kernels_read_plainly():
    src = _text()
    # the kernels' own loads and those of the functions that do their work
    for name in _early_kernels(src) + ['cdef_search_one', 'cdef_tile_filter', 'cdef_tile_item', 'upscale_item',
                                       'lr_tile_item', 'deblock_group']:
        params, body = _function(src, name)
        fixed = set(re.findall(r'const\s+\w+\s*\*\s*__restrict__\s+(\w+)', params))
        assert fixed <= PLANNED, (name, fixed - PLANNED)
        assert '__ldg' not in body, name


def test_grain_templates_run_beside_the_frame():
    """The templates depend on the frame's parameters only: forked off before the
    reconstruction, joined behind the filters."""
    src = re.sub(r'/\*.*?\*/|//[^\n]*', '', open(os.path.join(CSRC, 'decoder.cu')).read(), flags=re.S)
    body = _function(src, 'launch_step_plain')[1]
    order = ['cudaEventRecord(d->ev_fork, st)', 'cudaStreamWaitEvent(d->aux, d->ev_fork', 'launch_grain_template(',
             'cudaEventRecord(d->ev_join, d->aux)', 'launch_recon_stage(', 'launch_lr(',
             'cudaStreamWaitEvent(st, d->ev_join', 'launch_grain_blend(']
    at = [body.index(o) for o in order]
    assert at == sorted(at)
    assert re.search(r'launch_grain_template\([^;]*, d->aux\);', body)
