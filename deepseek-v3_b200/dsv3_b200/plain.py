"""Whether calling one of the host's modules does nothing but what a seam would do in its place.

A seam that computes several Linears in one launch does not call them.  That is the same only if their code is
``return linear(x, self.weight, self.bias, self.scale_fmt)`` (model.py:205; without the format in the parallel ones, :233 and
:262).  A name or a base class does not tell: adapter libraries call their classes ``Linear`` too, and a forward may be replaced on
the class.  So a class's code is run once on stand-ins that allow nothing else: ``linear``, ``weight``, ``bias`` and ``scale_fmt`` are
there, no builtins and no other names, attributes cannot be set, and code that catches exceptions is not looked at.  Code that
gets through, and returns what that one call of ``linear`` returned, has no effect but that call.

The answer is kept with the class, its two functions and their code, and found anew when one of them is another.
"""
from __future__ import annotations

import types

from torch.nn.modules import module as _nn_module

_Module = _nn_module.Module


class _Fixed(type):
    """A class whose attributes cannot be set, by way of an object's ``__class__``."""

    def __setattr__(cls, name, value):
        raise AttributeError(name)

    __delattr__ = __setattr__


class _Operand(metaclass=_Fixed):
    __slots__ = ()


class _Sealed(metaclass=_Fixed):
    """Attributes as given; none can be set."""

    def __init__(self, **attributes):
        self.__dict__.update(attributes)

    def __setattr__(self, name, value):
        raise AttributeError(name)

    __delattr__ = __setattr__


class _Call(metaclass=_Fixed):
    """Keeps the arguments of its calls and returns an operand."""
    __slots__ = ("calls", "result")

    def __init__(self):
        self.calls, self.result = [], _Operand()

    def __call__(self, x, weight, bias=None, scale_fmt=None):
        self.calls.append((x, weight, bias, scale_fmt))
        return self.result


def _sandboxed(function, model, stand_in):
    """``function`` with ``stand_in`` wherever it names ``model``, and nothing else of its surroundings."""
    if type(function) is not types.FunctionType:
        return None
    code = function.__code__
    if code.co_argcount != 2 or code.co_kwonlyargcount or code.co_flags & 0x2AC or getattr(code, "co_exceptiontable", b""):
        return None                                        # (0x2AC: *args, **kwargs, generators and coroutines)
    own = {"__builtins__": {}}
    if function.__globals__ is getattr(model, "__dict__", None):
        own.update(stand_in.__dict__)
    for name in code.co_names:
        if function.__globals__.get(name) is model:
            own[name] = stand_in
    cells = []
    for cell in function.__closure__ or ():
        try:
            if cell.cell_contents is not model:
                return None
        except ValueError:
            return None
        cells.append(types.CellType(stand_in))
    before = dict(own)
    inner = types.FunctionType(code, own, code.co_name, None, tuple(cells) or None)

    def run(self, x):
        y = inner(self, x)
        if own != before or any(c.cell_contents is not stand_in for c in cells):
            raise AttributeError("the surroundings were written to")
        return y

    return run


def _leads_to(value, model):
    """The model, as an attribute or in a list of its own."""
    return value is model or type(value) is list and len(value) == 1 and value[0] is model


def _links(module, model):
    return [name for name, value in getattr(module, "__dict__", {}).items() if _leads_to(value, model)]


def _run(module, model, target, **attributes):
    """Result of calling ``module`` in the sandbox, through its class's ``__call__`` and ``forward``; ``target`` stands for
    ``model.linear``, or for ``forward`` where it is None."""
    cls, x = type(module), _Operand()
    stand_in = _Sealed(**({"linear": target, "world_size": 1} if target else {}))
    for name in _links(module, model):
        attributes[name] = stand_in if module.__dict__[name] is model else (stand_in,)
    if target:
        run_forward = _sandboxed(getattr(cls, "forward", None), model, stand_in)
        if run_forward:
            attributes["forward"] = lambda x: run_forward(me, x)
    me = _Sealed(**attributes)
    before = dict(me.__dict__), dict(stand_in.__dict__)
    if cls.__call__ is _Module._wrapped_call_impl and cls._call_impl is _Module._call_impl:
        y = me.forward(x)
    else:
        run_call = _sandboxed(cls.__call__, model, stand_in)
        y = run_call(me, x) if run_call else None
    return (y, x) if before == (me.__dict__, stand_in.__dict__) else (None, x)


def _judge_linear(lin, model):
    takes_fmt = []
    for fmt in (None, "ue8m0"):
        linear, weight = _Call(), _Operand()
        y, x = _run(lin, model, linear, weight=weight, bias=None, scale_fmt=fmt)
        if y is not linear.result or len(linear.calls) != 1:
            return None
        got = linear.calls[0]
        if got[0] is not x or got[1] is not weight or got[2] is not None or got[3] not in (None, fmt):
            return None
        takes_fmt.append(got[3] is not None)
    return takes_fmt[1]


def _judge_mlp(mlp, model):
    result = _Operand()
    seen = []
    y, x = _run(mlp, model, None, forward=lambda x: (seen.append(x), result)[1])
    return True if y is result and len(seen) == 1 and seen[0] is x else None


_known = {}        # class -> (model, __call__, its code, forward, its code, attributes that lead to the model, answer)


def _answer(module, model, judge):
    """(attributes through which the module's code reaches the model, answer)"""
    cls = type(module)
    call, forward = cls.__call__, getattr(cls, "forward", None)
    known = _known.get(cls)
    if known is not None:
        of, call_, call_code, forward_, forward_code, found = known
        if (call is call_ and forward is forward_ and of is model and getattr(call, "__code__", None) is call_code
                and (forward is None or getattr(forward, "__code__", None) is forward_code)):
            return found
    try:
        found = _links(module, model), judge(module, model)
    except Exception:                                      # (what code does that the sandbox does not allow)
        found = (), None
    if len(_known) >= 64:
        _known.clear()
    _known[cls] = (model, call, getattr(call, "__code__", None), forward, getattr(forward, "__code__", None), found)
    return found


def linear_takes_fmt(lin, model, other=None):
    """Whether a call of ``lin`` hands its ``scale_fmt`` to ``model.linear``, where that is all it does while it has no bias and
    there is one rank; otherwise None.  ``other``: the same for another object of the class."""
    links, answer = _answer(lin, model, _judge_linear)
    for name in links:
        for one in (lin,) if other is None else (lin, other):
            if not _leads_to(one.__dict__.get(name), model):
                return None
    return answer


def calls_forward(mlp, model):
    """Whether a call of ``mlp`` is a call of its class's forward."""
    return _answer(mlp, model, _judge_mlp)[1] is not None


def installed_linear(model):
    """Whether ``model.linear`` is the function that install_linear made, and no wrapper that copied its attributes."""
    linear = getattr(model, "linear", None)
    return linear is not None and getattr(linear, "_dsv3_linear", None) is linear
