"""What a launch passes on: a number that a caller gives is taken as the integer it stands for, or refused. Without a GPU."""
import ast
from pathlib import Path

import numpy as np
import pytest
import torch

from scriptling_llm_lib_b200.csrc import bindings

SOURCE = Path(bindings.__file__).read_text()
CONVERTED = {"as_int", "c_int", "c_float", "c_longlong", "c_void_p", "_ptr"}


def _launches():
    """(function, argument) of every launch: the calls inside `_check(...)`, and the tuples of arguments that they unpack."""
    for fn in ast.walk(ast.parse(SOURCE)):
        if not isinstance(fn, ast.FunctionDef):
            continue
        for n in ast.walk(fn):
            if isinstance(n, ast.Call) and getattr(n.func, "id", "") == "_check" and isinstance(n.args[0], ast.Call):
                yield from ((fn, a) for a in n.args[0].args)
            if isinstance(n, ast.Assign) and getattr(n.targets[0], "id", "") in ("tail", "args"):
                yield from ((fn, a) for a in getattr(n.value, "elts", ()))


def test_no_launch_passes_a_callers_number_as_it_is():
    """ctypes takes a plain int only, turns None into 0 and a text into its address: what comes in through a parameter (sizes, windows,
    counts, or the step's) goes through `as_int`; what the wrapper reads off a tensor's shape is an int already."""
    plain, seen = [], 0
    for fn, arg in _launches():
        params = {a.arg for a in fn.args.args + fn.args.kwonlyargs} - {"self", "cls"}
        owned = {t.id for n in ast.walk(fn) if isinstance(n, ast.Assign) and isinstance(n.value, (ast.Attribute, ast.Tuple))
                 for t in ast.walk(n.targets[0]) if isinstance(t, ast.Name)}      # (M, K = a.shape)
        seen += 1
        if isinstance(arg, ast.Starred) or (isinstance(arg, ast.Call) and getattr(arg.func, "id", "") in CONVERTED):
            continue
        if isinstance(arg, (ast.Name, ast.BoolOp)):
            names = {n.id for n in ast.walk(arg) if isinstance(n, ast.Name)}
        elif isinstance(arg, ast.Attribute) or (isinstance(arg, ast.Call) and getattr(arg.func, "id", "") in ("max", "min")):
            names = {n.value.id for n in ast.walk(arg) if isinstance(n, ast.Attribute) and isinstance(n.value, ast.Name)}
        else:
            continue                                                               # sizes, literals, choices between them
        if names & (params - owned) and fn.name != "_run":                         # (_run: behind wrappers that read shapes)
            plain.append(f"{fn.name}: {ast.unparse(arg)}")
    assert seen > 1000 and not plain, plain


@pytest.mark.parametrize("value", [3, np.int64(3), np.uint8(3), torch.tensor(3), True])
def test_numbers_that_stand_for_integers(value):
    assert bindings.as_int(value) == int(value) and type(bindings.as_int(value)) is int


@pytest.mark.parametrize("value", [None, 3.0, "3", np.float32(3)])
def test_what_stands_for_no_integer_is_refused(value):
    with pytest.raises(TypeError):
        bindings.as_int(value)
