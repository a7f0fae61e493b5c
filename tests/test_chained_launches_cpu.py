"""Kernels that deal with other ranks never let the next launch of their stream start early, whatever that launch is."""

import os
import re

import pytest

import planmoe_b200

KERNELS = os.path.join(os.path.dirname(planmoe_b200.__file__), 'csrc', 'kernels')


def _bodies():
    for name in sorted(os.listdir(KERNELS)):
        if name.endswith('.cu'):
            text = open(os.path.join(KERNELS, name)).read()
            for m in re.finditer(r'__global__ void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\([^{;]*\{', text):
                depth, at = 1, m.end()
                while depth:
                    depth += {'{': 1, '}': -1}.get(text[at], 0)
                    at += 1
                yield name, m.group(1), text[m.end():at]


BODIES = {n: b for _, n, b in _bodies()}
WITH_OTHERS = [n for n, b in BODIES.items() if re.search(r'wait_flag_ge|copy_role|heap_bases', b)]


def test_found():
    assert {'gather_rows_kernel', 'grouped_gemm_kernel'} <= set(WITH_OTHERS) and 'local_gemm_kernel' not in WITH_OTHERS


@pytest.mark.parametrize('name', WITH_OTHERS)
def test_release_is_conditional(name):
    body = BODIES[name]
    assert 'chain_begin()' not in body
    for line in body.splitlines():
        if 'chain_release()' in line:
            assert re.match(r'\s*if \((w\.flags == nullptr|!COPY && alone\(p\))\) chain_release\(\);', line), line


@pytest.mark.parametrize('name', sorted(BODIES))
def test_wait_comes_first(name):
    """... and what is launched so waits before it lets anything go."""
    body = BODIES[name]
    if 'chain_release()' in body:
        assert body.index('chain_wait()') < body.index('chain_release()')
