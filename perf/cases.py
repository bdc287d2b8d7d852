"""The measured workloads: what a program that decodes with this framework has
it do, through its public entry points.

Three forms of call:

  planned  The split call of a pipelined player or transcoder: its planner
           threads have planned the frames ahead (Decoder.plan), the thread
           that drives the device queues each planned frame and its output
           (Decoder.decode_planned, then the NV12 pack into a device buffer,
           or the display planes) without waiting. A pass over inter frames
           is two successive frames of a running stream whose references are
           resident, the second predicting from the first; a pass over a key
           frame is that frame.
  whole    The direct call: a serialized frame in host memory in, planes or
           NV12 bytes in host memory out (Decoder.decode, Decoder.to_nv12).
  batch    The batched form: one planned frame of each of many independent
           streams a step (Batch.decode), at its default launch shape; a pass
           is two successive frame-sets.

Streams come from the seeded generator, so a case is the geometry, the bit
depth, the tools and the form; frames, motion, coefficients, filter levels and
film grain are drawn from the seed. All arithmetic of the path is integer, so
outputs are compared exactly.
"""
import ctypes
import os
from concurrent.futures import ThreadPoolExecutor

import torch

import av1ongpu_b200 as av1b

_TOOLS = {
    # intra modes, translation from one reference, deblocking and CDEF
    'basic': 0,
    # every tool but those of 'extended'
    'all': av1b.TOOLS_ALL,
    # every tool but restoration and film grain
    'no_output_filters': av1b.TOOLS_ALL & ~(av1b.TOOL_LR | av1b.TOOL_GRAIN),
    # inter-intra, intra block copy and raw residual blocks as well
    'extended': (av1b.TOOLS_ALL | av1b.TOOL_INTERINTRA | av1b.TOOL_INTRABC | av1b.TOOL_RESIDUAL),
}


def _single(name, call, picture, width, height, bit_depth, tools='all', coded_width=0, sb=64,
            output='nv12'):
    return {'name': name, 'call': call, 'picture': picture, 'width': width, 'height': height,
            'coded_width': coded_width, 'bit_depth': bit_depth, 'sb': sb, 'tools': tools,
            'output': output}


def _batch(name, n360, n720, n1080, n2160):
    return {'name': name, 'call': 'batch', 'n360': n360, 'n720': n720, 'n1080': n1080,
            'n2160': n2160}


def listed():
    return [
        # a thumbnail or preview stream: nothing but launches and latency
        _single('inter_240x136_10bit', 'planned', 'inter', 240, 136, 10),
        # the low rung of a streaming ladder
        _single('inter_640x360_8bit', 'planned', 'inter', 640, 360, 8),
        # a 720p 8-bit stream with the basic tools, and its key frame (a seek)
        _single('inter_1280x720_8bit_basic', 'planned', 'inter', 1280, 720, 8, 'basic'),
        _single('key_1280x720_8bit_basic', 'planned', 'key', 1280, 720, 8, 'basic'),
        # a picture whose sides are no multiple of a block, with the rarer tools
        _single('inter_1366x766_8bit_extended', 'planned', 'inter', 1366, 766, 8, 'extended', sb=128),
        # a 1080p 10-bit stream with every tool; its key frame shown as 16-bit planes
        _single('inter_1920x1080_10bit', 'planned', 'inter', 1920, 1080, 10),
        _single('key_1920x1080_10bit', 'planned', 'key', 1920, 1080, 10, output='planes'),
        # a 4K 10-bit stream coded at three quarters of its width (superres)
        _single('inter_2160p_superres_10bit', 'planned', 'inter', 3840, 2160, 10,
                coded_width=2880, sb=128),
        _single('key_2160p_superres_10bit', 'planned', 'key', 3840, 2160, 10,
                coded_width=2880, sb=128),
        # sixteen mixed streams decoded together
        _batch('batch_16_mixed_streams', 4, 6, 4, 2),
        # the direct call on host buffers, small and ordinary
        _single('whole_240x136_8bit', 'whole', 'inter', 240, 136, 8, output='nv12'),
        _single('whole_1920x1080_10bit', 'whole', 'inter', 1920, 1080, 10, output='planes'),
    ]


def _even(v):
    return max(16, int(round(v / 2)) * 2)


def draw(rng):
    form = rng.choices(['inter', 'key', 'whole', 'batch'], [11, 4, 2, 3])[0]
    if form == 'batch':
        n = [rng.randint(0, 4), rng.randint(0, 6), rng.randint(0, 4), rng.randint(0, 1)]
        if sum(n) < 2:
            n[0] += 2
        c = _batch('', *n)
        del c['name']
        return c
    top = 1080 if form == 'whole' else 2160
    height = _even(136 * (top / 136) ** rng.random())
    width = _even(height * rng.choice([16 / 9, 4 / 3, 2.0, 1.0, rng.uniform(0.6, 2.2)]))
    width = min(width, 3840)
    # a superres denominator of 9 to 16; 4K pictures are always coded narrower
    coded = 0
    if width * height > 2560 * 1600 or rng.random() < 0.25:
        coded = _even(width * 8 / rng.randint(11 if width * height > 2560 * 1600 else 9, 16))
    c = _single('', 'whole' if form == 'whole' else 'planned', 'key' if form == 'key' else 'inter',
                width, height, rng.choice([8, 8, 10, 10, 10, 12]),
                rng.choice(['basic', 'all', 'all', 'no_output_filters', 'extended']),
                coded, rng.choice([64, 64, 128]),
                rng.choice(['nv12', 'nv12', 'planes']))
    del c['name']
    return c


def _pitch(width):
    return (width + 63) // 64 * 64


def _frames(streams, counts, seed):
    """The first counts[i] frames of each stream (its generator arguments),
    generated on the host's cores."""
    jobs = [(i, k) for i in range(len(streams)) for k in range(counts[i])]

    def one(job):
        i, k = job
        w, h, cw, bd, sb, tools, refs = streams[i]
        return av1b.synth_frame_ex(w, h, cw, bd, sb, tools, seed * 64 + i, k, 0, max_refs=refs)

    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as ex:
        blobs = list(ex.map(one, jobs))
    out = [[] for _ in streams]
    for (i, _k), b in zip(jobs, blobs):
        out[i].append(b)
    return out


class _Device:
    """A plane in device memory for torch; it keeps its decoder alive."""

    def __init__(self, owner, ptr, rows, cols, stride):
        self.owner = owner
        # samples are at most 12 bits wide, so a signed 16-bit view holds them
        self.__cuda_array_interface__ = {'shape': (rows, cols), 'typestr': '<i2',
                                         'data': (ptr, False), 'strides': (2 * stride, 2),
                                         'version': 3}


class _Stream:
    """One stream: its decoder, its reference slots, the frames decoded
    before a pass and the planned frames (or host frames) of the pass."""

    def __init__(self, case, seed):
        self.case = case
        self.geometry = (case['width'], case['height'])
        tools = _TOOLS[case['tools']]
        key = case['picture'] == 'key'
        whole = case['call'] == 'whole'
        # frames decoded before the pass, frames of the pass
        before = 0 if key else 3
        n = 1 if key or whole else 2
        refs = 3 if tools & av1b.TOOL_COMPOUND else 1
        blobs = _frames([(case['width'], case['height'], case['coded_width'], case['bit_depth'],
                          case['sb'], tools, refs)], [before + n], seed)[0]
        self.dec = av1b.Decoder(0)
        self.slots = [self.dec.reserve_reference() for _ in range(before + n)]
        plans = []
        for k, b in enumerate(blobs):
            b.set_refs([self.slots[k - d] for d in b.get_refs()])
            if whole and k >= before:
                break
            p = self.dec.plan(b)
            if k < before:
                self.dec.decode_planned(p, slot=self.slots[k], wait=True)
                self.dec.free_plan(p)
            else:
                plans.append((p, self.slots[k]))
        self.plans = plans
        self.blob = blobs[-1] if whole else None
        self.pitch = _pitch(case['width'])
        size = av1b.nv12_size(case['width'], case['height'], 1, 1, self.pitch)
        self.nv12 = [torch.zeros(size, dtype=torch.uint8, device='cuda') for _ in range(n)]
        self.views = {}

    def planes(self, slot):
        """The planes of a slot's picture, where they are in device memory."""
        ptr = (ctypes.c_void_p * 3)()
        stride = (ctypes.c_int32 * 3)()
        if av1b.lib().av1b_slot_planes_device(self.dec.h, slot, ptr, stride):
            raise RuntimeError('slot_planes_device')
        at = (ptr[0], ptr[1], ptr[2])
        if at not in self.views:
            w, h = self.geometry
            self.views[at] = [torch.as_tensor(_Device(self.dec, ptr[p], rows, cols, stride[p]),
                                              device='cuda')
                              for p, (rows, cols) in enumerate(av1b.plane_shapes(w, h, 1, 1))]
        return self.views[at]

    def run_planned(self):
        shown = []
        for (plan, slot), nv12 in zip(self.plans, self.nv12):
            self.dec.decode_planned(plan, slot=slot, keep=True, wait=False)
            if self.case['output'] == 'nv12':
                self.dec.to_nv12_device(slot, self.pitch, nv12.data_ptr(), nv12.numel())
                shown.append(nv12)
            else:
                # the frame as it is shown; the next frame may reuse its planes
                shown = [self.planes(slot)]
        # the first frame's picture in its slot: what later frames predict from
        if len(self.plans) > 1:
            shown.append(self.planes(self.plans[0][1]))
        return shown

    def run_whole(self):
        if self.case['output'] == 'planes':
            slot, planes = self.dec.decode(self.blob, keep=True)
            self.dec.release_reference(slot)
            return planes
        slot, _ = self.dec.decode(self.blob, keep=True, read_back=False)
        out = self.dec.to_nv12(slot, self.pitch, *self.geometry)
        self.dec.release_reference(slot)
        return out


# the batched form's streams: width, height, bit depth by class
_CLASSES = (('n360', 640, 360, 8), ('n720', 1280, 720, 8), ('n1080', 1920, 1080, 10),
            ('n2160', 3840, 2160, 10))


def _batch_streams(case):
    return [(w, h, bd) for n, w, h, bd in _CLASSES for _ in range(case[n])]


class _Streams:
    """Many streams decoded as steps of one batch: two frame-sets before the
    pass, two in it."""

    def __init__(self, case, seed):
        geo = _batch_streams(case)
        n = len(geo)
        frames = _frames([(w, h, 0, bd, 64, av1b.TOOLS_ALL, 2) for w, h, bd in geo], [4] * n, seed)
        self.decs = [av1b.Decoder(0, planners=1, planner_threads=2) for _ in geo]
        slots = [[d.reserve_reference() for _ in range(4)] for d in self.decs]

        def plan(job):
            i, k = job
            b = frames[i][k]
            b.set_refs([slots[i][k - d] for d in b.get_refs()])
            return self.decs[i].plan(b)

        jobs = [(i, k) for k in range(4) for i in range(n)]
        with ThreadPoolExecutor(max_workers=min(n, os.cpu_count() or 1)) as ex:
            plans = list(ex.map(plan, jobs))
        self.plans = [plans[k * n:(k + 1) * n] for k in range(4)]
        self.slots = [[s[k] for s in slots] for k in range(4)]
        self.batch = av1b.Batch(0)
        for k in range(2):
            self.batch.decode(self.decs, self.plans[k], slots=self.slots[k])
        self.batch.sync()
        self.nv12 = []
        self.dst = []
        for _k in range(2):
            bufs = []
            for w, h, _bd in geo:
                size = av1b.nv12_size(w, h, 1, 1, _pitch(w))
                bufs.append(torch.zeros(size, dtype=torch.uint8, device='cuda'))
            self.nv12 += bufs
            self.dst.append([(t.data_ptr(), _pitch(g[0]), t.numel()) for t, g in zip(bufs, geo)])

    def run(self):
        for k in range(2):
            self.batch.decode(self.decs, self.plans[2 + k], slots=self.slots[2 + k],
                              nv12=self.dst[k])
        return self.nv12


def prepare(case, seed):
    s = _Streams(case, seed) if case['call'] == 'batch' else _Stream(case, seed)
    # the buffers' clearing is torch's work, on a stream the decoders do not wait for
    torch.cuda.synchronize()
    return s


def run(state):
    if isinstance(state, _Streams):
        return state.run()
    return state.run_whole() if state.blob is not None else state.run_planned()


def _frame_bytes(w, h, cw, inter, shown):
    """What one frame cannot do without: the coefficients (32 bits a coded
    sample), a sample of one reference for every predicted sample, the
    reconstructed picture, and the output."""
    coded, full = 1.5 * (cw or w) * h, 1.5 * w * h
    return 4 * coded + (2 * full if inter else 0) + 2 * full + shown


def work(case):
    if case['call'] == 'batch':
        b = sum(_frame_bytes(w, h, 0, True, 1.5 * w * h) for w, h, _bd in _batch_streams(case))
        return {'bytes': 2 * b, 'flops': 0}
    w, h = case['width'], case['height']
    # 8-bit NV12, or the 16-bit display planes
    shown = (1.5 if case['output'] == 'nv12' else 3) * w * h
    inter = case['picture'] == 'inter'
    n = 2 if inter and case['call'] == 'planned' else 1
    return {'bytes': n * _frame_bytes(w, h, case['coded_width'], inter, shown), 'flops': 0}


def tolerance(case):
    # integer arithmetic, specified sample for sample
    return 'exact'
