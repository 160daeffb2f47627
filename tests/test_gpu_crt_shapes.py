"""CRT at the counts where it changes between limb and digit kernels: 16 limb
lanes for few keys, 8 limb lanes up to a warp per scheduler, digits above."""
import pytest

from tests import test_gpu_digits as digits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half_bits,count", [(1536, 1), (1536, 592), (1536, 593), (1536, 1184), (1536, 1185), (2048, 1),
                                             (2048, 592), (2048, 593)])
def test_crt_between_shapes(handle, half_bits, count):
    digits.test_crt_digit_shapes(handle, half_bits, count)
