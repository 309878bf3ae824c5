import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN = os.path.join(ROOT, 'tests', 'golden')


def pytest_configure(config):
    config.addinivalue_line('markers', 'gpu: needs a CUDA device (run on a B200)')


def _has_gpu() -> bool:
    try:
        import torch

        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if _has_gpu():
        return
    skip = pytest.mark.skip(reason='no CUDA device')
    for item in items:
        if 'gpu' in item.keywords:
            item.add_marker(skip)


def seeded_weight(k: int, n: int, seed: int = 0, std: float = 0.02, dtype=np.float16) -> np.ndarray:
    """W ~ N(0, std^2), drawn in float32 and cast, as the benchmark configurations describe."""
    rng = np.random.default_rng(seed)
    return (rng.standard_normal((k, n), dtype=np.float32) * np.float32(std)).astype(dtype)


def seeded_activation(m: int, k: int, seed: int = 1, dtype=np.float16) -> np.ndarray:
    rng = np.random.default_rng(seed)
    return rng.standard_normal((m, k), dtype=np.float32).astype(dtype)


@pytest.fixture(scope='session')
def nvcc_library(tmp_path_factory):
    """Compiles a source of tests/cuda and loads it."""
    import ctypes
    import subprocess

    from hidet_b200 import build

    def load(source, *flags):
        out = str(tmp_path_factory.mktemp('cuda') / (source + '.so'))
        subprocess.check_call([build.find_nvcc(), *build.ARCH_FLAGS, '-O2', *flags, '-Xcompiler', '-fPIC', '-shared', os.path.join(ROOT, 'tests', 'cuda', source), '-o', out])
        return ctypes.CDLL(out)

    return load


@pytest.fixture(scope='session')
def large_kernels(nvcc_library):
    """tests/cuda/large_kernels.cu with the sources of the kernels that it calls."""
    import ctypes

    from hidet_b200 import build

    sources = [os.path.join(build.SRC_DIR, name + '.cu') for name in ('qlinear_pair', 'qlinear_mid', 'qlinear_prefill', 'qlinear_large', 'qlinear_decode', 'runtime')]
    lib = nvcc_library('large_kernels.cu', '-std=c++17', '-Xcompiler', '-fvisibility=hidden', '--threads', '0', *sources)
    p, i, n = ctypes.c_void_p, ctypes.c_int, ctypes.c_int64
    lib.plan.argtypes, lib.plan.restype = [n, n, n, i, p], None
    lib.small_plan.argtypes, lib.small_plan.restype = [n, n, n, p], None
    lib.launch.argtypes = [i, i, i, p, p, p, p, i, n, n, n, n, n, n, i, p, p, n, i, p]
    lib.launch_one_sm.argtypes = [p, p, p, p, i, n, n, n, n, n, p, ctypes.c_size_t, p]
    return lib


@pytest.fixture(scope='session')
def oracle_lib():
    import oracle

    return oracle
