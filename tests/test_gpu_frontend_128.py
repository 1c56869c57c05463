"""The fused front end of 128 points on either side of the filter count that chooses its kernel: bit for bit the four
calls."""
import pytest

from test_gpu_frontend import test_frontend_equals_plain_chain as equals_plain_chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [1, 2])
@pytest.mark.parametrize("window,hop", [(128, 32), (99, 50)])
@pytest.mark.parametrize("filters", [40, 200, 201])
def test_filters(gpu, filters, window, hop, power):
    equals_plain_chain(gpu, dict(nfft=128, window_length=window, window_step=hop, num_filter=filters, power=power))
