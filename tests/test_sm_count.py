"""How far ahead the kernels ask for memory follows the device's SM count (a
GB300's while no device is open), which the host writes into every program."""
import re

import pytest

import skelcl_gb300 as S


@pytest.mark.parametrize("kind,name,per_sm", [(S.KIND_SCAN, "SCL_SCAN_AHEAD", 1), (S.KIND_REDUCE, "SCL_REDUCE_AHEAD", 2)])
def test_distance_in_sms(built, kind, name, per_sm):
    src = S.generated_source(kind, "float func(float x, float y){ return x+y; }", ["float"], identity="0")
    sms = re.search(r"^#define SCL_SMS (\d+)$", src, re.M)
    assert sms and (int(sms.group(1)) == 152 or S.lib().scl_is_initialized())
    ahead = re.search(rf"^#define {name} (.*)$", src, re.M).group(1)
    assert eval(ahead, {"SCL_SMS": 1000}) == 1000 * per_sm
