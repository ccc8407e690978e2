"""The row limit of flow_linear_residual_noalloc: what it refuses, before any
CUDA call, and that the message gives the limit as the interface's own, not as
what the scratch (the same for any number of rows) would hold."""
import pytest


@pytest.mark.parametrize("nn", [0, -1, 262145, 2**31 - 1])
def test_refusal_names_the_interface_limit(nn):
    from flowgpu import capi
    with pytest.raises(capi.FlowError) as ei:
        capi.linear_residual_noalloc(32, 32, 32, 32, 32, nn, 0)
    msg = str(ei.value)
    assert f"nn = {nn} rows is outside 1..{capi.NOALLOC_MAX_ROWS}, the limit of the interface" in msg
    assert "scratch holds" not in msg
