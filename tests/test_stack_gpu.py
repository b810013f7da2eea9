"""The stack runner behind bench.py (rusty_b200/stack.py): what every output buffer holds after a step, against the
reference's arithmetic (dequantised f32 weights, f32 matmul), for both weight formats."""
import numpy as np
import pytest

from parity import TOL_FP32, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("native", [False, True])
@pytest.mark.parametrize("M", [1, 3])
def test_small_stack_outputs_match_the_reference_arithmetic(ctx, oracle, M, native):
    from rusty_b200 import DType
    from rusty_b200.stack import LinearStack
    from rusty_b200.workloads import StackShape
    shape = StackShape("tiny", d=256, q=256, kv=128, ffn=640, vocab=1024, layers=2)
    st = LinearStack(ctx, shape, M, DType.FP32, DType.FP32, seed=3, native=native, keep_host=True)
    assert st.native == native and not st.swiglu
    if native:
        assert set(st.plans()) == {"gemv_mma"}   # K % 128 == 0 everywhere: the re-laid-out affine format
    st.step()
    ctx.sync()
    # buffers are reused from layer to layer: each one holds the output of the LAST Linear that wrote it
    last = {}
    for i, (name, y) in enumerate(zip(st.names, st._ys)):
        last[id(y)] = i
    assert len(last) >= 4
    for i in last.values():
        x = st.host_inputs[st.dims[i][1]]
        ref = oracle.matmul_bt(x, st.host_wf[i], mt=True)
        got = np.frombuffer(st._ys[i].to_bytes(ctx), np.float32).reshape(M, st.out_n[i])
        assert rel_err(got, ref) <= TOL_FP32, st.names[i]


@pytest.mark.parametrize("native", [False, True])
@pytest.mark.parametrize("M", [1, 2, 3])
def test_stack_with_norms_under_capture(ctx, oracle, M, native):
    """The step with the blocks' norms, recorded and replayed: at few rows, and in the native format, the norm is a kernel of its
    own whose output needs a buffer, and nothing can be allocated while a capture is open."""
    from rusty_b200 import DType
    from rusty_b200.stack import LinearStack
    from rusty_b200.workloads import StackShape
    # (a width no other test uses: the pool must not happen to hold such a buffer)
    st = LinearStack(ctx, StackShape("tiny", d=320, q=256, kv=64, ffn=640, vocab=1024, layers=2), M, DType.FP32, DType.FP32, seed=4, swiglu=True,
                     norms=True, native=native, keep_host=True)
    graph = st.capture()
    graph.launch()
    ctx.sync()
    x, w = st.host_inputs[320], st.norm_w[-1].to_vec(ctx)
    got = np.frombuffer(st.logits.to_bytes(ctx), np.float32).reshape(M, 1024)
    assert rel_err(got, oracle.matmul_bt(oracle.rms_norm(x, w), st.host_wf[-1], mt=True)) <= TOL_FP32
