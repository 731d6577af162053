"""How the prefill GEMM divides a call (iq_qmm_plan, host code only): scratch that serves every smaller call."""
import itertools

import pytest

from ingot_b200 import capi

SMS = 148
FORMATS = [(4, 64, 0), (8, 64, 0), (4, 32, 0), (4, 32, capi.IQ_MODE_MXFP4), (2, 128, 0)]


def plan(n, k, fmt, rows, gate_up=False, sms=SMS):
    bits, group, mode = fmt
    return capi.qmm_plan(n, k, bits, group, rows, mode, gate_up, sms)


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("gate_up", [False, True])
def test_scratch_for_the_most_rows_serves_all_calls(fmt, gate_up):
    """A call's partial sums fit what a call of any larger number of rows asks for (the split of a call alone is no measure: 4096 x 14336
    takes 20 MB at 512 rows and none at 640), and that never falls."""
    if gate_up and fmt[0] == 2:
        pytest.skip("ternary gate/up is two kernels")
    widths = [64, 192, 1024, 2048, 2880, 4096, 7744, 14336, 50048]
    falls = 0
    for n, k, sms in itertools.product(widths, [128, 1024, 2048, 5120, 14336], [SMS, 146, 132, 75]):
        asked = last = 0
        for rows in itertools.chain([17, 33, 50], range(64, 2049, 64), [3072, 4096, 8192]):
            p = plan(2 * n if gate_up else n, k, fmt, rows, gate_up, sms)
            assert p.split_bytes <= p.bytes_up_to_rows, (n, k, sms, rows)
            assert p.bytes_up_to_rows >= asked, (n, k, sms, rows)
            falls += p.split_bytes < last
            asked, last = p.bytes_up_to_rows, p.split_bytes
        assert asked <= 2 * sms * 192 * 128 * 4 + 256  # two slots of 192 tokens per SM
    assert falls > 0  # what the bound is for
