"""Sizes at which a launch's grid or a block's memory ends, on the GPU."""
import os
import subprocess

import numpy as np
import pytest

from pypercolate_gb300 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from pypercolate_gb300 import _native as nat
    nat.lib_handle()
    return nat


# 262,136: the last number of probabilities whose tiles of 8, two blocks each,
# fit the grid's y; 524,280: the last that the entry point takes
@pytest.mark.parametrize('P', [262136, 262137, 300000, 524280])
@pytest.mark.parametrize('model', ['bond', 'site'])
def test_many_probabilities(gpu, P, model):
    """Every p of a long grid gets its canonical averages: those of the same
    values of p in an ensemble of few (same runs, same bits, whatever the
    tiles' probabilities)."""
    from pypercolate_gb300.ensemble import Ensemble
    ps = np.linspace(0.05, 0.95, P)
    ens = Ensemble('chain', 5, ps, precision='fp32', micro=False, model=model)
    ens.run(130, key=3)
    mean, m2 = (t.cpu().numpy().reshape(P, 7) for t in (ens.mean, ens.m2))
    for first in (0, P // 2 // 8 * 8, P - 16 - P % 8):
        few = Ensemble('chain', 5, ps[first:first + 16], precision='fp32', micro=False, model=model)
        few.run(130, key=3)
        for a, b in ((mean, few.mean), (m2, few.m2)):
            assert np.array_equal(a[first:first + 16], b.cpu().numpy().reshape(16, 7))


@pytest.mark.parametrize('what', ['runs', 'permutations'])
def test_threads_with_blocks_of_different_memory(gpu, what):
    """Two host threads on streams of their own launch one kernel with much and
    with little shared memory per block: neither takes the other's away."""
    import threading

    import torch
    from pypercolate_gb300 import hpc
    lib = gpu.lib_handle()
    failed = []

    def runs(L, stream, times):
        spec = hpc.GraphSpec(gpu.GRAPH_GRID2D, L)
        g, rec = spec.struct(), gpu.Records(spec.M + 1, 1, with_edge=False)
        need = lib.nz_microcanonical_workspace_bytes(g, 1, gpu.PERM_PHILOX)
        ws = gpu.device_empty(need)
        for _ in range(times):
            if lib.nz_microcanonical(g, 1, 1, gpu.PERM_PHILOX, 1, 0, None, None, None, 1, gpu.ptr(ws), need,
                                     rec.struct(), stream.cuda_stream):
                failed.append(L)
        stream.synchronize()

    def permutations(M, stream, times):
        words, lens = (torch.zeros(1, dtype=torch.int32, device='cuda') for _ in range(2))
        out = torch.empty(M, dtype=torch.int32, device='cuda')
        torch.cuda.synchronize()
        for _ in range(times):
            if lib.nz_permutations(M, 1, gpu.PERM_MT19937, 0, 0, gpu.ptr(words), gpu.ptr(lens), 1, gpu.ptr(out),
                                   stream.cuda_stream):
                failed.append(M)
        stream.synchronize()

    work, sizes = {'runs': (runs, (256, 181)), 'permutations': (permutations, (65160, 30000))}[what]
    threads = [threading.Thread(target=work, args=(size, torch.cuda.Stream(), 1500)) for size in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


def test_a_launch_that_fails_leaves_no_error_behind(gpu, tmp_path):
    """What a launch returns, for a block or a shared-memory limit that the host
    refuses, is not found again by the next call's check."""
    source = tmp_path / 'refused.cu'
    source.write_text('''
#include <cstdio>
#include "nz_internal.cuh"
__global__ void nothing() {}
int main() {
    const bool block = nz::launch_kernel(nothing, dim3(1), 4096, 0, 0, nullptr) != cudaSuccess;
    const bool limit = nz::launch_kernel(nothing, dim3(1), 32, 0, 1 << 30, nullptr) != cudaSuccess;
    printf("%d %d %d\\n", block, limit, (int)cudaPeekAtLastError());
}
''')
    program = str(tmp_path / 'refused')
    subprocess.run([build.nvcc(), *build.ARCH, '-std=c++17', '--expt-relaxed-constexpr', '-I', build.CSRC, '-I',
                    os.path.join(os.path.dirname(build.HERE), 'include'), '-o', program, str(source)], check=True)
    assert subprocess.run([program], check=True, capture_output=True, text=True).stdout.split() == ['1', '1', '0']
