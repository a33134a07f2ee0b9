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


def test_the_extension_is_this_interpreters_and_this_torchs(recipe):
    import sysconfig
    import torch
    from q8_kernels_b200 import _host
    assert os.path.realpath(_host.__file__) == os.path.realpath(recipe.HOST_PATH)
    assert recipe.HOST_PATH.endswith(sysconfig.get_config_var("EXT_SUFFIX")) and not os.path.exists(os.path.join(recipe.PKG_DIR, "_host.so"))
    assert torch.__version__.startswith(_host.__torch_version__)


@pytest.mark.parametrize("key", ["this", "another", None])
def test_another_torch_needs_another_extension(recipe, monkeypatch, tmp_path, key):
    """What the extension was built against is kept beside the objects; file times say nothing about it (an older torch put in
    place later).  torch's own C++ ABI is passed on."""
    torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
    this = torch_dir + "\n" + open(os.path.join(torch_dir, "version.py")).read()
    recipe.HOST_KEY = str(tmp_path / "key")
    if key is not None:
        (tmp_path / "key").write_text(this if key == "this" else this.replace("__version__ = '", "__version__ = '0."))
    recipe.OBJ_DIR, recipe.PKG_DIR = str(tmp_path), str(tmp_path)
    ran = []

    class Done:
        returncode, stdout, stderr = 0, "1\n", ""

    monkeypatch.setattr(recipe.subprocess, "run", lambda cmd, **k: ran.append(cmd) or Done)
    monkeypatch.setattr(recipe, "_stale", lambda *a: False)
    recipe._build_host(False)
    compiled = [c for c in ran if c[0] == "g++"]
    assert len(compiled) == (key != "this")
    assert all("-D_GLIBCXX_USE_CXX11_ABI=1" in c and recipe.HOST_PATH in c for c in compiled)
    assert (tmp_path / "key").read_text() == this
