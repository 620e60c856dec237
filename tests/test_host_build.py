"""The host-call extension is tied to one Python and one torch: its name and its build record say so, and an import that does not fit
is explained."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def build(lib_built):
    import importlib.util
    spec = importlib.util.spec_from_file_location("minit_b200_build_copy", os.path.join(ROOT, "minit_b200", "csrc", "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_another_torch_makes_it_stale(build, monkeypatch):
    import sysconfig
    import torch
    from minit_b200 import _lib
    assert build.HOST.endswith("_host" + sysconfig.get_config_var("EXT_SUFFIX"))
    assert _lib._host.torch_version == torch.__version__ == build.torch_version()
    assert build.host_is_current()
    monkeypatch.setattr(build, "torch_version", lambda: "0.0")
    assert not build.host_is_current()


@pytest.mark.parametrize("stub,words", [(None, "missing or does not load"), ("", "missing or does not load"),
                                        ("torch_version = '1.0'", "was built for torch 1.0")])
def test_an_import_that_does_not_fit_is_explained(build, tmp_path, stub, words):
    """A package without the extension, with one that is no extension of this build, and with one of another torch."""
    pkg = tmp_path / "minit_b200"
    shutil.copytree(os.path.join(ROOT, "minit_b200"), pkg, ignore=shutil.ignore_patterns("_host*", "csrc", "__pycache__", "*.so"))
    os.symlink(build.LIB, pkg / "libminit_b200.so")
    if stub is not None:
        (pkg / "_host.py").write_text(stub)
    r = subprocess.run([sys.executable, "-c", "import minit_b200"], cwd=tmp_path, capture_output=True, text=True, env={**os.environ, "PYTHONPATH": str(tmp_path)})
    assert r.returncode != 0 and words in r.stderr and "minit_b200/csrc/build.py" in r.stderr, r.stderr[-800:]
