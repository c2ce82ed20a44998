"""What the native call path does with arguments that it refuses and with the errors of what it calls: a Python error each, the one
that names the cause, and no other. Nothing is launched, so no GPU is needed."""
import pytest

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def capi():
    import nnforge_b200.capi as capi
    return capi


class StreamAddress:
    """What int() makes a stream's address of."""

    def __int__(self):
        return 0


class BrokenStream:
    @property
    def cuda_stream(self):
        raise LookupError("no stream today")


@pytest.mark.parametrize("stream", [0, StreamAddress()])
def test_a_refused_argument_keeps_its_error(capi, stream):
    """The first refusal is what the caller hears of, whatever kind of argument comes after it."""
    x = torch.zeros(2, 4, 6, 6)                       # not on a device
    for f in (lambda: capi.softmax_fwd(x, x, stream=stream),
              lambda: capi.add_fwd(x, [x, x], stream=stream),
              lambda: capi.nll_bwd(x, x, x, None, "not a number", stream=stream),
              lambda: capi.bn_infer_act(0, x, (x, x, x, x), acts=[capi.relu()], stream=stream),
              lambda: capi.maxpool_fwd(0, 0, x, capi.pool((2, 2), (2, 2)), stream=stream),
              lambda: capi.apply_gradient([{"data": x, "gradient": x, "learning_rate": 0.1}], stream=stream)):
        with pytest.raises(AssertionError, match="contiguous CUDA tensors"):
            f()
    with pytest.raises(KeyError, match="learning_rate"):
        capi.apply_gradient([{"data": 0, "gradient": 0}], stream=stream)
    with pytest.raises(TypeError):
        capi.apply_gradient([], momentum="much", stream=stream)


def test_errors_of_the_stream_are_its_own(capi):
    with pytest.raises(LookupError, match="no stream today"):
        capi.apply_gradient([], stream=BrokenStream())
    with pytest.raises(TypeError):
        capi.apply_gradient([], stream="0x0 or so".split)


def test_an_empty_step_is_no_error(capi):
    capi.apply_gradient([], stream=0)
    capi.apply_gradient((), stream=StreamAddress())
