"""What the native call path does with arguments that it refuses and with the errors of what it calls: a Python error each, the one
that names the cause, and no other. Nothing is launched, so no GPU is needed; where no device must be found, the calls are made in a
process that sees none."""
import collections
import os
import subprocess
import sys
import types

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

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


def test_a_chunk_is_any_mapping(capi):
    """A chunk that is not a plain dict is asked through its own item and get: it gets as far as the check of its tensors."""
    x = torch.zeros(4)                                # not on a device
    full = {"data": x, "gradient": x, "learning_rate": 0.1, "weight_decay": 0.0}
    for chunk in (types.MappingProxyType(full), collections.UserDict(full), collections.OrderedDict(full),
                  collections.defaultdict(lambda: 0.1, data=x, gradient=x)):
        with pytest.raises(AssertionError, match="contiguous CUDA tensors"):
            capi.apply_gradient([chunk], stream=0)
    for chunk in ({"data": x, "gradient": x}, types.MappingProxyType({"data": x, "gradient": x})):
        with pytest.raises(KeyError, match="learning_rate"):
            capi.apply_gradient([chunk], stream=0)
    with pytest.raises(TypeError):
        capi.apply_gradient([x.numpy], stream=0)


class Likeness:
    """Answers what a tensor is asked, without being one."""

    def __init__(self, *shape, cuda=True, address=0):
        self.shape, self.is_cuda, self.address, self.asked = shape, cuda, address, 0

    def is_contiguous(self):
        return True

    def data_ptr(self):
        self.asked += 1
        return self.address

    def numel(self):
        return 24

    def element_size(self):
        return 4


def test_what_answers_as_a_tensor_is_taken_as_one(capi):
    """The library itself refuses these for their null addresses, after every argument has been read."""
    x, ws = Likeness(2, 3, 2, 2), Likeness(24)
    for f in (lambda: capi.softmax_fwd(x, x, stream=0),
              lambda: capi.add_fwd(x, [x, x], stream=0),
              lambda: capi.add_bwd(x, x, stream=0),
              lambda: capi.maxpool_fwd(x, x, x, capi.pool((2, 2), (2, 2)), stream=0),
              lambda: capi.bn_train_fwd(x, x, x, x, x, x, 1e-5, workspace=ws, stream=0),
              lambda: capi.apply_gradient([{"data": x, "gradient": x, "learning_rate": 0.1}], stream=0)):
        x.asked = 0
        with pytest.raises(capi.NnfError, match="null|has no data"):
            f()
        assert x.asked >= 2
    with pytest.raises(AssertionError, match="contiguous CUDA tensors"):
        capi.softmax_fwd(x, Likeness(2, 3, cuda=False), stream=0)
    with pytest.raises(AttributeError):
        capi.softmax_fwd(x, object(), stream=0)


def test_structures_are_of_their_own_type(capi):
    """24 bytes of anything else are no activation: they would hold an address that nobody gave."""
    import ctypes
    x = Likeness(2, 3, 2, 2)
    for wrong in (bytes(ctypes.sizeof(capi.Act)), capi.pool((2, 2), (2, 2)), "tanh"):
        with pytest.raises(TypeError):
            capi.act_fwd(x, x, wrong, stream=0)
        with pytest.raises(TypeError):
            capi.bn_infer_act(x, x, acts=[wrong], stream=0)
    for wrong in (bytes(ctypes.sizeof(capi.Pool)), capi.relu()):
        with pytest.raises(TypeError):
            capi.maxpool_fwd(x, x, x, wrong, stream=0)


def test_extents_that_do_not_suffice(capi):
    """As indexing and unpacking a shape report them."""
    with pytest.raises(IndexError):
        capi.softmax_fwd(0, Likeness(6), stream=0)
    with pytest.raises(ValueError):
        capi.maxpool_fwd(0, 0, Likeness(6, 4, 4), capi.pool((2, 2), (2, 2)), stream=0)


def test_errors_of_torch_are_python_errors():
    """No device, a tensor without storage: errors that a program can catch, from the functions and from the layer objects."""
    code = """
import torch
import nnforge_b200.capi as capi, nnforge_b200.host as host
x = torch.zeros(2, 4)
sparse = x.to_sparse()
tester, updater = host.Tester("TanH", 4, 1, 1), host.Updater("TanH", 4, 1, 1)
for f in (lambda: capi.softmax_fwd(x, x),
          lambda: capi.apply_gradient([]),
          lambda: tester.enqueue_forward_propagation(x, [], [x], 2),
          lambda: updater.enqueue_forward_propagation(x, [], [x], 2),
          lambda: tester.enqueue_forward_propagation(sparse, [], [x], 2),
          lambda: tester.enqueue_forward_propagation(x, [], [sparse], 2)):
    try:
        f()
        print("none")
    except RuntimeError:
        print("caught")
"""
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, CUDA_VISIBLE_DEVICES=""), capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, "exit status %d\n%s" % (p.returncode, p.stderr[-2000:])
    assert p.stdout.split() == ["caught"] * 6
