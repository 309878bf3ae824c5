"""The quotient in the epilogues' SiLU against the division and against 64 bits."""
import ctypes
import struct

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def compare(nvcc_library):
    f = nvcc_library('silu.cu', '-std=c++17').compare
    f.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]

    def run(begin, step, count, errors):
        out = torch.zeros(6, dtype=torch.int64, device='cuda')
        assert f(begin, step, count, errors, out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        return out.tolist()

    return run


def _bits(x):
    return struct.unpack('I', struct.pack('f', x))[0]


# every float of the binades in which exp(-g) and 1 meet, and a part of those around them: where one vanishes against the other, where exp(-g)
# overflows, up to gates that no sum reaches
@pytest.mark.parametrize('low,high,step', [(2.0 ** -100, 2.0 ** -30, 31), (2.0 ** -30, 0.03125, 5), (0.03125, 32.0, 1), (32.0, 87.0, 1), (87.0, 128.0, 1), (128.0, 2.0 ** 125, 61)])
@pytest.mark.parametrize('sign', [0, 0x80000000])
def test_quotient_of_the_division(compare, low, high, step, sign):
    count = (_bits(high) - _bits(low)) // step + 1
    differ, apart, worst, worst_here, total, total_here = compare(_bits(low) | sign, step, count, high <= 87.0)
    # The reciprocal and the product are off by at most 1 + 1/2 ulp, a relative 2^-22.4, and the correction by no more than that part and a rounding of
    # itself, 2^-44 of the quotient.  Among quotients spread evenly over an ulp, 2^-24 of the value or more, that moves at most 2 * 2^-44 / 2^-24
    # over a rounding boundary, two in a million, each to the next float.
    assert apart <= 1 and differ <= 2e-6 * count + 8
    # Against 64 bits: one ulp more for those few at most, which is not to be seen in the mean.
    assert worst_here <= worst + 1000 * (differ > 0) and total_here <= total + 1000 * differ


@pytest.mark.parametrize('gate', [0.0, -0.0, float('inf'), float('-inf'), float('nan')])
def test_quotient_of_zeros_infinities_and_nan(compare, gate):
    assert compare(_bits(gate), 0, 1, False)[:2] == [0, 0]
