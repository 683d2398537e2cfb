"""Element types that the Reduce/Zip AllPairs compiles for (no device)."""
import pytest

import skelcl_gb300 as S


def compile_pairs(left, right):
    S.compile_only(S.KIND_ALLPAIRS, "float func(float x, float y){ return x+y; }", [left, right, "float"],
                   source2=f"float func({left} x, {right} y){{ return 1; }}", identity="0")


@pytest.mark.parametrize("t", ["char", "unsigned char", "short", "int", "long", "float", "double"])
def test_scalar_operands(built, t):
    compile_pairs(t, "float")
    compile_pairs("double", t)


@pytest.mark.parametrize("t", ["float2", "float4", "int2", "double2"])
def test_vector_operands_refused(built, t):
    """Vector types do not sit on their own size, which the kernel's copies
    into shared memory want."""
    for pair in ((t, "float"), ("float", t), (t, t)):
        with pytest.raises(S.SclError) as e:
            compile_pairs(*pair)
        assert e.value.status == S.ERR_COMPILE
