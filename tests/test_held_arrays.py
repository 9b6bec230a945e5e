"""The check that a kept table of addresses still belongs to an ensemble's tensors (CPU)."""
import os
import subprocess
import sys
from array import array

import pytest
import torch

import legateboost_b200 as lb  # noqa: F401
from legateboost_b200.tree import _holds, _holds_in_python

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


class Model:
    def __init__(self):
        self.leaf_value, self.feature, self.split_value = torch.zeros(7, 1), torch.zeros(7, dtype=torch.int32), torch.zeros(7)


def _table(models):
    source = tuple(t for m in models for t in (m.leaf_value, m.feature, m.split_value))
    return source, array("q", [t.data_ptr() for t in source]).tobytes()


def test_holds_the_same_tensors_where_they_were():
    models = [Model() for _ in range(5)]
    source, at = _table(models)
    assert _holds(models, source, at) and _holds(list(models), source, at) and _holds([], (), b"")
    models[3].leaf_value.fill_(2.0)  # contents do not matter
    assert _holds(models, source, at)
    assert not _holds(models[:4], source, at) and not _holds(models + [Model()], source, at)
    assert not _holds([models[1], models[0]] + models[2:], source, at)


@pytest.mark.parametrize("name", ["leaf_value", "feature", "split_value"])
def test_another_or_a_moved_tensor_is_seen(name):
    models = [Model() for _ in range(3)]
    source, at = _table(models)
    was = getattr(models[2], name)
    setattr(models[2], name, was.clone())
    assert not _holds(models, source, at)
    setattr(models[2], name, None)
    assert not _holds(models, source, at)
    setattr(models[2], name, was)
    assert _holds(models, source, at)
    was.data = was.clone()  # the same object elsewhere
    assert not _holds(models, source, at)


def test_errors_are_python_errors():
    models = [Model()]
    source, at = _table(models)
    with pytest.raises(TypeError):
        _holds(models, list(source), at)
    with pytest.raises(ValueError):
        _holds(models, source, at[:-1])
    del models[0].feature
    with pytest.raises(AttributeError):
        _holds(models, source, at)

    class Odd(Model):  # an attribute that changes the list while it is walked
        @property
        def feature(self):
            models.clear()
            return None

        @feature.setter
        def feature(self, value):
            pass

    models[:] = [Odd(), Model()]
    assert not _holds(models, source + source, at + at)


def test_another_torch_or_python_has_a_module_of_its_own():
    """What is compiled in are the layouts of one torch and one Python: a module of another pair neither counts as built nor is
    ever loaded."""
    import sysconfig

    from legateboost_b200 import build

    assert _holds.__module__ == "legateboost_b200." + build.module_name()
    other = build.module_path("0.1.0+none")
    assert build.module_path() != other and not os.path.exists(other) and os.path.exists(build.module_path())
    assert build.module_path().endswith(sysconfig.get_config_var("EXT_SUFFIX")) and build.module_name("0.1.0+none").isidentifier()


@pytest.mark.parametrize("n", [1, 4])
def test_the_python_way_gives_the_same_answers(n):
    def changed(models, what):
        last = models[-1]
        if what == "shorter":
            return models[:-1]
        if what == "longer":
            return models + [Model()]
        if what == "order":
            return models[::-1]
        if what == "none":
            last.feature = None
        elif what == "other":
            last.split_value = last.split_value.clone()
        elif what == "moved":
            last.leaf_value.data = last.leaf_value.clone()
        elif what == "filled":
            last.leaf_value.fill_(3.0)
        return models

    for what in ("same", "shorter", "longer", "order", "none", "other", "moved", "filled"):
        models = [Model() for _ in range(n)]
        source, at = _table(models)
        models = changed(models, what)
        answer = _holds_in_python(models, source, at)
        assert answer == _holds(models, source, at) == (what in ("same", "filled") or (what == "order" and n == 1)), what
    with pytest.raises(AttributeError):
        _holds_in_python([object()], source[:3], at[:24])


def test_without_the_module_tables_are_checked_all_the_same():
    """The module makes the check faster; without it (not built, or built for another torch) predictions work as with it."""
    program = """
import importlib.util, sys
spec = importlib.util.spec_from_file_location("lbk_build", sys.argv[1])
build = importlib.util.module_from_spec(spec)
spec.loader.exec_module(build)
sys.modules["legateboost_b200." + build.module_name()] = None  # importing it is an ImportError
import torch
from legateboost_b200 import tree
assert tree._holds is tree._holds_in_python
class Model:
    def __init__(self):
        self.leaf_value, self.feature, self.split_value = torch.zeros(7, 1, dtype=torch.float64), -torch.ones(7, dtype=torch.int32), torch.zeros(7, dtype=torch.float64)
models = [Model() for _ in range(3)]
table = tree.TreeTable([(m.leaf_value, m.feature, m.split_value) for m in models])
assert table.matches(models) and table.matches(tuple(models)) and not table.matches(models[:2])
models[1].feature = models[1].feature.clone()
assert not table.matches(models)
"""
    subprocess.run([sys.executable, "-c", program, os.path.join(ROOT, "legate-boost_b200", "build.py")], check=True, cwd=ROOT)
