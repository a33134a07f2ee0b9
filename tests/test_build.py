"""CPU checks of the build recipe: what it needs, and when it builds again.  Nothing is compiled here."""
import importlib.util
import os

import pytest

import helpers as Hp


@pytest.fixture
def recipe():
    spec = importlib.util.spec_from_file_location("q8k_build_recipe", os.path.join(Hp.REPO_ROOT, "q8_kernels_b200", "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("options", [{}, {"library_only": True}])
def test_the_library_needs_no_torch(recipe, monkeypatch, capsys, options):
    """The C ABI is built for programs without Python too: a machine without torch leaves out the extension and says so."""
    find = importlib.util.find_spec
    monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
    monkeypatch.setattr(recipe, "_stale", lambda *a: False)
    assert recipe.build(**options) == recipe.LIB_PATH
    assert ("torch is not installed" in capsys.readouterr().err) == (not options)
