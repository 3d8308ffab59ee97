"""Rules of the kernels' sources that no run shows reliably: what a launch that
begins before the one in front of it has ended may promise the compiler."""

import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, 'chainerkfac_b200', 'csrc')

# What a plan or a call writes once, from the host or by a launch that is over
# before any of its early launches begins.
STATIC = {'MatInfo', 'RefineItem', 'GemmDesc', 'PackRows', 'GradSizes',
          'RunParams'}


def source():
    text = ''
    for path in sorted(glob.glob(os.path.join(CSRC, '*.cu*'))):
        text += re.sub(r'//[^\n]*', '', open(path).read()) + '\n'
    return text


def closing(text, start, pair):
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError('unbalanced')


def functions(text):
    """{name: (is a kernel, parameters, body)} of the device functions."""
    found = {}
    for m in re.finditer(r'__global__|__device__', text):
        head = re.compile(r'(?!__launch_bounds__\b)\b(\w+)\s*\(')
        at = m.end()
        bounds = re.match(r'[^;{]*?__launch_bounds__\s*\(', text[at:])
        if bounds:
            at = closing(text, at + bounds.end() - 1, '()') + 1
        name = head.search(text, at)
        if not name or re.search(r'[;{}=]', text[at:name.start()]):
            continue
        end = closing(text, name.end() - 1, '()')
        brace = re.match(r'\s*\{', text[end + 1:])
        if not brace:
            continue
        start = end + brace.end()
        found[name.group(1)] = (m.group() == '__global__',
                                text[name.end():end],
                                text[start:closing(text, start, '{}')])
    return found


@pytest.fixture(scope='module')
def early():
    """The kernels that wait for the launch in front themselves."""
    fns = functions(source())
    waits = {'wait_for_launch_before'}
    while True:
        more = {n for n, (_, _, body) in fns.items()
                if any(re.search(r'\b%s\s*\(' % w, body) for w in waits)}
        if more <= waits:
            break
        waits |= more
    return {n: fns[n] for n in waits if n in fns and fns[n][0]}


def test_early_kernels_are_found(early):
    assert {'damp_copy_kernel', 'chol_diag_kernel', 'panel_solve_kernel',
            'refine_gate_kernel', 'refine_apply_kernel', 'packed_tile_kernel',
            'pack_rows_kernel', 'tc_tile_kernel'} <= set(early)


def test_early_kernels_promise_nothing_of_what_others_write(early):
    """`__restrict__` lets the compiler read ahead of the wait, whatever stands
    between (and through a cache that nothing keeps up to date): only for tables
    that stay as they are from the first launch to the last."""
    for name, (_, params, body) in early.items():
        for p in params.split(','):
            if '__restrict__' in p:
                m = re.match(r'\s*const\s+(\w+)\s*\*\s*__restrict__\s+\w+\s*$', p)
                assert m and m.group(1) in STATIC, (name, p.strip())
        assert not re.search(r'__ldg\s*\(|ld\.global\.nc', body), name


def test_tensor_memory_goes_back_behind_what_is_under_way():
    """Where a bounded wait has run out, copies and MMAs may still be under way:
    only tc_release hands tensor memory back, which gives them time, and only
    behind the block's last barrier, where the flag is everybody's."""
    text = source()
    assert text.count('tcgen05.dealloc') == 1
    fns = functions(text)
    assert 'tcgen05.dealloc' in fns['tc_release'][2]
    assert '__nanosleep' in fns['tc_release'][2]
    users = 0
    for name, (kernel, _, body) in fns.items():
        if 'tc_release(' not in body:
            continue
        users += 1
        assert kernel, name
        last = body[body.rindex('__syncthreads()'):]
        assert re.search(r'tc_release\([^;]*abort_flag != 0\)', last), name
        assert 'tcgen05.mma' not in last and 'complete_tx' not in last, name
    # (the allocation of the diagonal kernel is in a function of its own)
    assert users == len([b for _, _, b in fns.values()
                         if 'tcgen05.alloc' in b])
