"""Rules of order between kernels and copies, read from the sources.

``launch_pdl`` lets a grid come up during the last wave of the one before it,
and callers' streams are not ordered with the default one.  A broken rule shows
on the GPU only as a hang or a wrong value that depends on timing, so the rules
are read from the sources: these tests need no GPU.
"""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    'dinosaur_b200', 'csrc')


def source(path):
  with open(path) as f:
    text = f.read()
  text = re.sub(r'/\*.*?\*/', ' ', text, flags=re.S)
  return re.sub(r'//[^\n]*', ' ', text)


SOURCES = {os.path.basename(p): source(p)
           for p in sorted(glob.glob(os.path.join(CSRC, '*.cu*')))}


def closing(text, start, pair):
  """Index just past the bracket that closes text[start]."""
  depth = 0
  for i in range(start, len(text)):
    depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
    if depth == 0:
      return i + 1
  raise ValueError('unbalanced')


def kernels():
  """{name: (parameter list, body)} of every __global__ function."""
  out = {}
  for text in SOURCES.values():
    for match in re.finditer(r'__global__\s+void\s+(?:__launch_bounds__\s*\()?', text):
      i = match.end()
      if match.group().rstrip().endswith('('):
        i = closing(text, i - 1, '()')
      name = re.compile(r'\s*(\w+)\s*\(').match(text, i)
      end = closing(text, name.end() - 1, '()')
      brace = text.index('{', end)
      out[name.group(1)] = (text[name.end():end - 1], text[brace:closing(text, brace, '{}')])
  return out


KERNELS = kernels()
DEPENDENT = sorted(k for k, (_, body) in KERNELS.items() if 'pdl_' in body)


def test_the_kernels_are_found():
  assert {'legendre_tc_kernel', 'legendre_forward_simt', 'rfft_inverse_kernel',
          'pe_nodal_hybrid_kernel', 'swe_stage_kernel'} <= set(DEPENDENT)


TENSOR_MEMORY = sorted(k for k, (_, body) in KERNELS.items() if 'tcgen05.alloc' in body)


@pytest.mark.parametrize('name', TENSOR_MEMORY)
def test_dependents_start_only_after_tensor_memory_is_held(name):
  # A dependent CTA allocates tensor memory before it waits for its predecessor.
  # If a CTA of the predecessor could still have to allocate then, the dependent
  # could take the columns it needs and each would wait for the other for good.
  _, body = KERNELS[name]
  # Paths that return early hold no tensor memory.
  body = re.sub(r'\{[^{}]*\breturn\s*;[^{}]*\}', ' ', body)
  assert body.count('pdl_trigger()') == 1
  before = body[:body.index('pdl_trigger()')]
  # One thread's trigger counts for its CTA: the CTA's barrier lies between.
  assert 'tcgen05.alloc' in before
  assert '__syncthreads()' in before[before.index('tcgen05.alloc'):]


@pytest.mark.parametrize('name', DEPENDENT)
def test_every_dependent_kernel_waits(name):
  # On every path: once at least, and before each early return.
  _, body = KERNELS[name]
  assert 'pdl_wait()' in body
  first = body.index('pdl_wait()')
  for match in re.finditer(r'\breturn\s*;', body):
    assert match.start() > first, name
  for match in re.finditer(r'\{([^{}]*)\breturn\s*;[^{}]*\}', body):
    if match.start() < body.rindex('pdl_wait()'):
      assert 'pdl_wait()' in match.group(1), name


# Plan tables: written once when the plan is made, before any launch of these kernels.
TABLES = {'ptab', 'ptab_off', 'tw_n', 'tw_i', 'wq', 'f'}


@pytest.mark.parametrize('name', DEPENDENT)
def test_earlier_results_are_not_declared_read_only(name):
  # A const __restrict__ pointer says that nothing writes what it points to while
  # the kernel runs, and lets its loads move over the wait; the predecessor may
  # still be writing then.
  parameters, _ = KERNELS[name]
  read_only = re.findall(r'const\s+\w+\s*\*\s*__restrict__\s+(\w+)', parameters)
  assert set(read_only) <= TABLES, name


def test_no_read_only_loads():
  # __ldg and ld.global.nc make the same promise wherever they are called.
  for name, text in SOURCES.items():
    assert '__ldg' not in text and 'ld.global.nc' not in text, name
    for match in re.finditer(r'__device__[^;{]*?\(([^)]*)\)\s*\{', text):
      assert not re.search(r'const[^,]*\*\s*__restrict__', match.group(1)), name


def test_uploads_are_finished_before_they_return():
  # A copy from pageable host memory may return while its last part is still on
  # its way, and kernels on a caller's non-blocking stream do not wait for the
  # default stream.  So every upload goes through upload(), which waits.
  copies = {name: text.count('cudaMemcpyHostToDevice') for name, text in SOURCES.items()}
  assert {k: v for k, v in copies.items() if v} == {'dino_internal.cuh': 1}
  text = SOURCES['dino_internal.cuh']
  start = text.index('{', text.index('int upload('))
  body = text[start:closing(text, start, '{}')]
  assert body.index('cudaMemcpyHostToDevice') < body.index('cudaStreamSynchronize')


def test_launch_rules_ask_the_device_for_its_multiprocessors():
  for name, text in SOURCES.items():
    assert not re.search(r'\b148\b', text), name
