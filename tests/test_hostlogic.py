"""Host-side shape logic against the reference's known answers."""
import numpy as np
import pytest

from theano_b200 import hostlogic as H
from theano_b200 import shim


def test_output_shape_known_answers():
    # TestGetConvOutShape.test_basic, reference test_abstract_conv.py:102-118
    x, w, sub, dil = (3, 2, 12, 9), (4, 2, 5, 6), (1, 2), (2, 1)
    assert H.forward_shape(x, w, "valid", sub, dil)[0] == (3, 4, 4, 2)
    assert H.forward_shape(x, w, "half", sub, dil)[0] == (3, 4, 12, 5)
    assert H.forward_shape(x, w, "full", sub, dil)[0] == (3, 4, 20, 7)
    assert H.forward_shape(x, w, (1, 2), sub, dil)[0] == (3, 4, 6, 4)


def test_border_mode_normalisation():
    assert H.normalize_border_mode(2) == ((2, 2), (2, 2))
    assert H.normalize_border_mode((1, (2, 3))) == ((1, 1), (2, 3))
    assert H.normalize_border_mode("half") == "half"
    for bad in (-1, (1,), (1, -2), "same", ((1, 2, 3), 1)):
        with pytest.raises(ValueError):
            H.normalize_border_mode(bad)


def test_gradient_shape_inference():
    # stride 1: both sizes can be inferred; stride 2 / half: they must be given (corr.py:286-294)
    assert H.gradweights_kshape((2, 3, 9, 9), (2, 4, 7, 7), "valid", (1, 1), (1, 1)) == (3, 3)
    assert H.gradweights_kshape((2, 3, 9, 9), (2, 4, 11, 11), "full", (1, 1), (1, 1)) == (3, 3)
    assert H.gradweights_kshape((2, 3, 9, 9), (2, 4, 5, 5), (0, 0), (1, 1), (2, 2)) == (3, 3)
    with pytest.raises(ValueError):
        H.gradweights_kshape((2, 3, 9, 9), (2, 4, 4, 4), "valid", (2, 2), (1, 1))
    with pytest.raises(ValueError):
        H.gradweights_kshape((2, 3, 9, 9), (2, 4, 9, 9), "half", (1, 1), (1, 1))
    assert H.gradinputs_imshape((4, 3, 3, 3), (2, 4, 7, 7), "valid", (1, 1), (1, 1))[0] == (9, 9)
    with pytest.raises(ValueError):
        H.gradinputs_imshape((4, 3, 3, 3), (2, 4, 4, 4), "valid", (2, 2), (1, 1))


def test_inconsistent_shapes_raise_value_error():
    # reference test_abstract_conv.py:602-656: output shapes the forward cannot produce
    for o in (-3, -1, 1, 2):
        pads = H.resolve_pads("valid", (3, 3), (1, 1))
        with pytest.raises(ValueError):
            H.check_consistent((1, 1, 7, 7), (1, 1, 3, 3), (1, 1, 5 + o, 5 + o), pads, (1, 1), (1, 1), 1)
    with pytest.raises(ValueError):
        H.forward_shape((1, 3, 5, 5), (2, 2, 3, 3), "valid", (1, 1), (1, 1))
    with pytest.raises(ValueError):
        H.forward_shape((1, 3, 5, 5), (2, 3, 7, 7), "valid", (1, 1), (1, 1))
    with pytest.raises(TypeError):
        H.forward_shape((1, 3, 5), (2, 3, 3, 3), "valid", (1, 1), (1, 1))


def _plan(border_mode="valid", subsample=(1, 1), dilation=(1, 1), groups=1):
    return shim._plans.find(shim._plan_forward, "fwd", (2, 4, 9, 9), (6, 4 // groups, 3, 3), border_mode, subsample, dilation,
                            groups, True, np.dtype(np.float32))


@pytest.mark.parametrize("options", [dict(border_mode=1.0), dict(border_mode=(1.0, 1)), dict(subsample=(2.0, 2.0)),
                                     dict(dilation=(1.0, 1))], ids=lambda d: str(d).replace(" ", ""))
def test_what_is_refused_does_not_depend_on_calls_before(options):
    """Floats that equal integers have the same hash: a plan made for the integers must not answer for them."""
    whole = {k: tuple(int(e) for e in v) if isinstance(v, tuple) else int(v) for k, v in options.items()}
    def answer(**o):
        try:
            return [type(n) for n in _plan(**o)[0]]         # float strides give a float shape, which no array takes
        except (ValueError, TypeError) as e:
            return type(e)
    shim._plans.clear()
    refused = answer(**options)
    assert refused != [int] * 4
    for _ in range(2):
        shape, desc = _plan(**whole)
        assert [type(n) for n in shape] == [int] * 4 and _plan(**whole)[1] is desc
        assert answer(**options) == refused


def test_plans_are_found_again_for_equal_arguments():
    first = _plan(border_mode=((1, 2), (2, 1)), subsample=(2, 1))
    assert _plan(border_mode=tuple([tuple([1, 2]), tuple([2, 1])]), subsample=tuple([2, 1])) is first
    assert _plan(border_mode=((1, 2), (2, 1)), subsample=(np.int64(2), np.int64(1)))[0] == first[0]
    assert _plan(border_mode=[[1, 2], [2, 1]], subsample=[2, 1])[0] == first[0]              # lists: worked out each time
