"""Every part names the kernel files it may launch (they are built before the first step): the names are compared with what the launchers
that the part's code refers to load, found in the source."""
import ast
import importlib
import inspect
import os
import pkgutil

import pytest
import torch

import turboquant_cpp_b200 as tq
from turboquant_cpp_b200 import kernels, parts
from turboquant_cpp_b200.parts.base import Part

PACKAGE = tq.__name__


def _aliases(tree, package):
    """Local name -> (module of kernels, function or None), from a module's imports."""
    out = {}
    for node in ast.walk(tree):
        if not isinstance(node, ast.ImportFrom):
            continue
        base = package.split(".")[:len(package.split(".")) - node.level + 1] if node.level else []
        module = ".".join(base + ([node.module] if node.module else []))
        for a in node.names:
            if module == PACKAGE + ".kernels":
                out[a.asname or a.name] = (a.name, None)
            elif module.startswith(PACKAGE + ".kernels."):
                out[a.asname or a.name] = (module.rsplit(".", 1)[1], a.name)
    return out


def _referred(node, aliases):
    """(module, function) of the launchers that a piece of code mentions."""
    for n in ast.walk(node):
        if isinstance(n, ast.Attribute) and isinstance(n.value, ast.Name) and aliases.get(n.value.id, (None, 0))[1] is None and n.value.id in aliases:
            yield aliases[n.value.id][0], n.attr
        elif isinstance(n, ast.Name) and n.id in aliases and aliases[n.id][1] is not None:
            yield aliases[n.id]


def _launchers():
    """(module, function) -> the libraries it loads, its callees' included."""
    loads, calls = {}, {}
    for info in pkgutil.iter_modules(kernels.__path__):
        with open(os.path.join(kernels.__path__[0], info.name + ".py"), encoding="utf-8") as f:
            tree = ast.parse(f.read())
        constants = {t.id: n.value.value for n in tree.body if isinstance(n, ast.Assign) and isinstance(n.value, ast.Constant) for t in n.targets
                     if isinstance(t, ast.Name)}
        aliases = _aliases(tree, PACKAGE + ".kernels")
        functions = [n for n in tree.body if isinstance(n, ast.FunctionDef)]
        for f in functions:
            key = (info.name, f.name)
            loads[key] = {(a.value if isinstance(a, ast.Constant) else constants.get(getattr(a, "id", None))) for n in ast.walk(f)
                          if isinstance(n, ast.Call) and getattr(n.func, "id", "") == "load_kernel" for a in n.args} - {None}
            calls[key] = set(_referred(f, aliases)) | {(info.name, g.name) for g in functions for n in ast.walk(f) if isinstance(n, ast.Name) and n.id == g.name}
    for _ in range(6):
        for key, callees in calls.items():
            for c in callees:
                loads[key] = loads[key] | loads.get(c, set())
    return loads


LAUNCHERS = _launchers()


def _parts():
    for info in pkgutil.iter_modules(parts.__path__):
        module = importlib.import_module(f"{PACKAGE}.parts.{info.name}")
        for _, cls in inspect.getmembers(module, inspect.isclass):
            if cls.__module__ == module.__name__ and issubclass(cls, Part) and "kernels" in cls.__dict__ and not info.name == "block":
                yield module, cls


class _Branch:
    def kernels(self):
        return ["gemm_f32"]


def _named(cls, dtype, bound=None):
    """What a part of sizes of 64 names, its weights not bound yet or of `bound`."""
    sized = type("Sized", (cls,), {"__getattr__": lambda self, name: 64})
    part = sized.__new__(sized)
    part.run_dtype, part.left, part.right, part.w13 = dtype, _Branch(), _Branch(), None
    if bound is not None:
        part.w_any = torch.zeros((2, 64), dtype=bound)
    return set(part.kernels())


@pytest.mark.parametrize("module,cls", list(_parts()), ids=lambda x: getattr(x, "__name__", str(x)).split(".")[-1])
def test_a_part_names_what_it_may_launch(module, cls):
    tree = ast.parse(inspect.getsource(module))
    aliases = _aliases(tree, module.__package__)
    body = next(n for n in ast.walk(tree) if isinstance(n, ast.ClassDef) and n.name == cls.__name__)
    helpers = [n for n in tree.body if isinstance(n, ast.FunctionDef) and any(isinstance(m, ast.Name) and m.id == n.name for m in ast.walk(body))]
    libraries = set()
    for code in [body] + helpers:
        for target in _referred(code, aliases):
            libraries |= LAUNCHERS.get(target, set())
    either = _named(cls, torch.float32) | _named(cls, torch.bfloat16)
    missing = libraries - either
    assert not missing, f"{cls.__name__} launches {sorted(missing)} without naming them"
    if "gemm_f32" in libraries:
        # a checkpoint's float32 weights stay float32 in a bfloat16 run: named once they are bound
        assert "gemm_f32" in _named(cls, torch.float32) and "gemm_f32" in _named(cls, torch.bfloat16, torch.float32)


def test_a_bfloat16_run_builds_no_float32_product():
    from turboquant_cpp_b200.parts.attention import AttentionMixer
    assert "gemm_f32" not in _named(AttentionMixer, torch.bfloat16, torch.bfloat16) | _named(AttentionMixer, torch.bfloat16)


def test_the_launchers_are_found():
    assert LAUNCHERS["recurrence", "delta_chunks"] == {"ssm", "delta_chunks"} and LAUNCHERS["linear", "linear"] == {"gemm_f32"}
    assert LAUNCHERS["attention", "attention_tiled"] == {"attention", "attention_f32"} and len(list(_parts())) >= 15
