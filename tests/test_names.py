"""Every global name that the package's functions use exists: a name that nothing defines shows only when its line runs, and
the measurement programs' commands run in no other test."""
import builtins
import dis
import importlib
import pkgutil
import types

import pytest

import torchinferno_b200

MODULES = sorted(m.name for m in pkgutil.walk_packages(torchinferno_b200.__path__, "torchinferno_b200.") if not m.name.endswith("__main__"))


def _undefined(code: types.CodeType, known: set[str]) -> list[str]:
    found = [f"{code.co_name}: {i.argval}" for i in dis.get_instructions(code) if i.opname == "LOAD_GLOBAL" and i.argval not in known]
    for const in code.co_consts:
        if isinstance(const, types.CodeType):
            found += _undefined(const, known)
    return found


@pytest.mark.parametrize("name", MODULES)
def test_every_global_name_is_defined(name):
    module = importlib.import_module(name)
    with open(module.__file__) as source:
        code = compile(source.read(), module.__file__, "exec")
    assert not _undefined(code, set(vars(module)) | set(dir(builtins)))
