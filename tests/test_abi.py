"""The C ABI (include/vesta_b200.h, libvesta_b200.so): loads without a GPU, exports every declared
symbol, reports errors through its status + message convention. No GPU compute here."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, 'include', 'vesta_b200.h')).read()
    text = re.sub(r'/\*.*?\*/', '', text, flags=re.S)
    return sorted(set(re.findall(r'\b(vesta_\w+)\s*\(', text)))


def test_header_declares_the_launch_path():
    names = declared_symbols()
    for need in ('vesta_nvrtc_compile', 'vesta_module_load', 'vesta_module_get_function',
                 'vesta_func_set_max_dynamic_smem', 'vesta_occupancy', 'vesta_launch_cooperative',
                 'vesta_step_bind', 'vesta_step_run', 'vesta_last_error'):
        assert need in names


def test_library_exports_every_declared_symbol(built_library):
    lib = ctypes.CDLL(str(built_library))
    for name in declared_symbols():
        assert hasattr(lib, name), name
    assert lib.vesta_rt_version() == 1


def test_error_convention(built_library):
    from vesta_gpu_b200 import launch
    L = launch.lib()
    mod = ctypes.c_void_p()
    assert L.vesta_module_load(None, ctypes.byref(mod)) != 0
    assert b'null' in L.vesta_last_error()
    with pytest.raises(RuntimeError):
        launch.ok(L.vesta_step_run(None, None, 1))
    bound = ctypes.c_void_p()
    assert L.vesta_step_bind(None, 1, 1, 0, 0, None, ctypes.byref(bound)) != 0


def test_nvrtc_through_the_abi_without_a_gpu(built_library):
    from vesta_gpu_b200 import launch
    cubin = launch.compile_cubin('extern "C" __global__ void k(float* p) { p[threadIdx.x] = 1.f; }', cache=False)
    assert cubin[:4] == b'\x7fELF'
    with pytest.raises(RuntimeError) as err:
        launch.compile_cubin('extern "C" __global__ void k(float* p) { p[0] = undefined_name; }', cache=False)
    assert 'undefined_name' in str(err.value)          # the compiler log is in the message (vesta/launch.py:21-24)


def test_step_kernel_compiles_for_sm_100a(built_library):
    from vesta_gpu_b200 import launch
    from vesta_gpu_b200.build import lower_for
    from vesta_gpu_b200.shapes import TINY
    for kw in (dict(), dict(per_sequence_t=True), dict(timing=1), dict(feedback=False)):
        low = lower_for(TINY, 3, 17, **kw)
        assert launch.compile_cubin(low.src, cache=False)[:4] == b'\x7fELF'


def test_no_cpu_path():
    """without a CUDA device the product refuses to run instead of falling back"""
    import torch
    if torch.cuda.is_available():
        pytest.skip('a GPU is present')
    from vesta_gpu_b200.launch import Kernel
    from vesta_gpu_b200.build import lower_for
    from vesta_gpu_b200.shapes import TINY
    with pytest.raises(RuntimeError):
        Kernel(lower_for(TINY, 1, 8))


def test_product_does_not_import_the_oracle():
    pkg = os.path.join(ROOT, 'vesta_gpu_b200')
    for dirpath, _, files in os.walk(pkg):
        for f in files:
            if f.endswith(('.py', '.cuh', '.cpp', '.cu')):
                text = open(os.path.join(dirpath, f), encoding='utf-8').read()
                assert 'import oracle' not in text and 'from oracle' not in text, f


def test_static_step_refuses_oversized_requests_before_touching_the_gpu(built_library):
    """vesta_step_static checks its sizes on the host first: more residues than its argument array holds, a scratch
    size whose byte count would wrap around, and output ranges outside the scratch are all refused with a message
    (no CUDA call has been made at that point, so this runs without a GPU)"""
    lib = ctypes.CDLL(str(built_library))
    lib.vesta_static_last_error.restype = ctypes.c_char_p
    sz, vp, ull = ctypes.c_size_t, ctypes.c_void_p, ctypes.c_ulonglong
    ptrs = (ull * 64)(*([0x1000] * 64))
    fn = vp(0x10)                                   # never launched: every case below is refused before that

    def call(n_res=20, scratch=1024, counters=64, lo=0, ln=16, no=16, nn=4):
        return lib.vesta_step_static(fn, 148, 288, 0, n_res, ptrs, ull(0), ull(0), ull(0), sz(scratch), sz(counters),
                                     sz(lo), sz(ln), vp(None), sz(no), sz(nn), vp(None), vp(None), vp(None))
    assert call(n_res=57) != 0 and b'residues' in lib.vesta_static_last_error()
    assert call(n_res=-1) != 0
    assert call(scratch=(1 << 62) + 8) != 0 and b'static scratch holds' in lib.vesta_static_last_error()
    assert call(scratch=(4 << 20) // 4) != 0 and b'static scratch holds' in lib.vesta_static_last_error()
    assert call(counters=1 << 20) != 0 and b'counter' in lib.vesta_static_last_error()
    assert call(lo=(1 << 64) - 8, ln=16) != 0 and b'output range' in lib.vesta_static_last_error()
    assert call(no=1000, nn=100) != 0 and b'output range' in lib.vesta_static_last_error()


def pass_desc(**kw):
    """a descriptor of a pass that would be accepted, over addresses that nobody follows"""
    from vesta_gpu_b200.passes import Desc, _PTRS
    d = Desc(L=2, D=128, H=2, F=256, N=211, tmax=64, cpos=64, rows=16, logit_rows=16, eps=1e-5, scale=8.0)
    for n in _PTRS:
        setattr(d, n, 0x10000)
    for n, v in kw.items():
        setattr(d, n, v)
    return d


def create_pass(d, workspace=0x10000):
    """-> the message with which vesta_pass_create refuses (without a GPU every descriptor is refused in the end)"""
    from vesta_gpu_b200 import launch
    L, out = launch.lib(), ctypes.c_void_p()
    assert L.vesta_pass_create(ctypes.byref(d), ctypes.c_void_p(workspace), 0, ctypes.byref(out)) != 0 and not out.value
    return L.vesta_last_error().decode()


def test_a_pass_refuses_tensors_that_its_loads_cannot_reach(built_library):
    for name in ('keys', 'vals', 'wte', 'qkvw', 'ow', 'fcw', 'pw'):
        assert '16-byte boundary' in create_pass(pass_desc(**{name: 0x10008})), name
    for name in ('wpe', 'ln1w', 'ln1b', 'ln2w', 'ln2b', 'lnfw', 'lnfb'):
        assert '8-byte boundary' in create_pass(pass_desc(**{name: 0x10002})), name
    for name in ('x', 't', 'logits', 'bar', 'qkvb', 'ob', 'fcb', 'pb'):
        assert 'missing' in create_pass(pass_desc(**{name: None})), name
    few = dict(exact=2, rows=4, logit_rows=4)
    for name in ('ob', 'pb'):                       # (a step from packed weights reads these four elements at a time)
        for off in (2, 4):
            assert '8-byte boundary' in create_pass(pass_desc(**few, **{name: 0x10000 + off})), name
    assert '256-byte boundary' in create_pass(pass_desc(), workspace=0x10010)


def test_a_pass_refuses_sizes_that_would_leave_its_buffers(built_library):
    """fewer logit rows than prompts that can end in a pass (metadata and logits would be written past their ends), counts below
    zero or beyond what 32-bit indices hold, empty dimensions"""
    from vesta_gpu_b200 import launch
    L, n = launch.lib(), ctypes.c_size_t()

    def sizes(**kw):
        d = pass_desc(**kw)
        return L.vesta_pass_workspace(ctypes.byref(d), ctypes.byref(n))
    assert sizes() == 0 and sizes(prompts=4, rows=64, logit_rows=4) == 0 and sizes(prompts=40, rows=16, logit_rows=16) == 0
    for bad in (dict(prompts=4, rows=64, logit_rows=3), dict(prompts=40, rows=16, logit_rows=15), dict(prompts=-1), dict(logit_rows=17), dict(rows=0),
                dict(rows=2 ** 31 - 1), dict(D=0, H=0), dict(F=0), dict(F=-16), dict(tmax=0), dict(cpos=0), dict(exact=1, rows=17, logit_rows=17)):
        assert sizes(**bad) != 0 and L.vesta_last_error().startswith(b'vesta_pass'), bad


def test_a_step_from_packed_weights_refuses_what_it_is_not_written_for(built_library):
    """fewer logit rows than rows (its end writes a row of logits and a token for every row, past the ends of both), one row and more
    than four, wide rows, an MLP of more than 32 features per SM, prompts"""
    from vesta_gpu_b200 import launch
    L, n = launch.lib(), ctypes.c_size_t()
    for rows, lrows, fine in ((4, 4, True), (4, 3, False), (2, 2, True), (2, 1, False)):
        d = pass_desc(exact=2, rows=rows, logit_rows=lrows)
        assert (L.vesta_pass_workspace(ctypes.byref(d), ctypes.byref(n)) == 0) == fine, (rows, lrows)
        if not fine:
            assert b'packed weights' in L.vesta_last_error() and 'packed weights' in create_pass(d)
    for kw in (dict(rows=1, logit_rows=1), dict(rows=5, logit_rows=5), dict(rows=8, logit_rows=8), dict(rows=9, logit_rows=9), dict(D=1088, H=17), dict(F=4752),
               dict(prompts=4)):
        d = pass_desc(**dict(dict(exact=2, rows=4, logit_rows=4), **kw))
        assert L.vesta_pass_workspace(ctypes.byref(d), ctypes.byref(n)) != 0 and b'packed weights' in L.vesta_last_error(), kw


@pytest.mark.parametrize('name,exact', [('gpt2', 0), ('gpt2_xl', 0), ('tiny3', 0), ('heads20', 0), ('gpt2', 1), ('tiny', 1)])
def test_tiles_of_a_pass_fit_a_block(built_library, name, exact):
    """every tile that is chosen is one the kernels are written for: the rows of one product, the columns of tensor memory (two
    accumulators), shared memory, no empty part of a fold; rows at fp32 accuracy in one tile of head and remainder"""
    from vesta_gpu_b200.passes import tiles
    from vesta_gpu_b200.shapes import SHAPES
    sh = SHAPES[name]
    for rows in ([1, 3, 8, 9, 16] if exact else [1, 15, 16, 17, 23, 64, 65, 100, 128, 129, 256, 1000, 1024, 4097, 9200, 16384]):
        lrows = min(rows, 256)
        d = pass_desc(L=sh.L, D=sh.D, H=sh.H, F=sh.F, N=sh.N, rows=rows, logit_rows=lrows, exact=exact, prompts=0 if exact else lrows)
        for kind, (bm, bn, stages, parts, smem) in tiles(d, rows, lrows).items():
            at, blocks = (name, rows, kind), (-(-sh.F // 64) if kind == 'p2' else sh.D // 64)
            assert bm in (64, 128, 256) and bn % 16 == 0 and 16 <= bn <= (64 if bm == 64 else 256), at
            assert stages >= 1 and smem <= 227 * 1024, at
            assert 1 <= parts <= (12 if kind in ('proj', 'p2') else 1) and -(-blocks // -(-blocks // parts)) == parts, at
            assert bm != 256 or (bn >= 64 and kind != 'logits'), at
            if exact:
                assert (bm, bn) == (64, 2 * (8 if rows <= 8 else 16)), at


def test_blocks_of_a_steps_projection_that_keep_others_away(built_library):
    """what vesta_pass_tiles reports is what a block is launched with: more than its stages where there is a block for about every SM
    and three would fit one; not for few blocks or wide rows"""
    from vesta_gpu_b200.passes import tiles
    from vesta_gpu_b200.shapes import SHAPES
    for name, rows, prompts, more in (('gpt2', 64, 0, True), ('gpt2', 37, 0, True), ('gpt2', 23, 0, False), ('gpt2_xl', 16, 0, False),
                                      ('gpt2_xl', 64, 0, False), ('heads20', 16, 0, False), ('gpt2', 77, 1, True), ('gpt2_xl', 77, 1, False)):
        sh = SHAPES[name]
        d = pass_desc(L=sh.L, D=sh.D, H=sh.H, F=sh.F, N=sh.N, rows=rows, logit_rows=prompts or rows, prompts=prompts)
        bm, bn, stages, parts, smem = tiles(d, rows, d.logit_rows)['proj']
        assert (smem == 110 * 1024) == more, (name, rows, prompts, bm, bn, stages, parts, smem)
