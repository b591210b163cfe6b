"""The build step: what counts as out of date.  Works on files of its own in place of the sources and outputs; no compiler runs."""
import importlib.util
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """build.py on a small tree: two CUDA sources, a header, the host module's source, the public header; everything built at time 1000, objects
    left behind later than the outputs (the compilers run at the same time)."""
    spec = importlib.util.spec_from_file_location("_lo_build_under_test", os.path.join(ROOT, "lightop_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    pkg = tmp_path / "pkg"
    (pkg / "csrc").mkdir(parents=True)
    (tmp_path / "include").mkdir()
    files = {"a.cu": pkg / "csrc" / "a.cu", "b.cu": pkg / "csrc" / "b.cu", "common.h": pkg / "csrc" / "common.h", "host.cpp": pkg / "csrc" / "host.cpp",
             "lightop_b200.h": tmp_path / "include" / "lightop_b200.h", "a.o": pkg / "csrc" / "a.o", "lib": pkg / "lib.so", "host": pkg / "_host.so"}
    for name, path in files.items():
        path.write_text("")
        t = {"lib": 1001, "host": 1000, "a.o": 2000}.get(name, 900)
        os.utime(path, (t, t))
    for name, value in dict(HERE=str(pkg), CSRC=str(pkg / "csrc"), LIB=str(files["lib"]), HOST=str(files["host"]), SOURCES=["a.cu", "b.cu"]).items():
        monkeypatch.setattr(build, name, value)
    monkeypatch.setattr(build, "built_for", lambda: "torch 1, Python x")
    build.really_possible = build.host_possible
    monkeypatch.setattr(build, "host_possible", lambda: True)
    files["host"].write_bytes(b"..[built for torch 1, Python x]..")
    os.utime(files["host"], (1000, 1000))
    return build, files


def test_a_finished_build_is_up_to_date(tree):
    build, _ = tree
    assert not build.needs_build()


@pytest.mark.parametrize("name,lib,host", [("b.cu", True, False), ("common.h", True, False), ("host.cpp", False, True), ("lightop_b200.h", True, True),
                                           ("a.o", False, False)])
def test_each_output_has_its_own_sources(tree, name, lib, host):
    build, files = tree
    os.utime(files[name], (3000, 3000))
    assert build.outdated() == [p for p, old in ((build.LIB, lib), (build.HOST, host)) if old]
    assert build.needs_build() == (lib or host)


@pytest.mark.parametrize("name", ["lib", "host"])
def test_a_missing_output_is_built(tree, name):
    build, files = tree
    files[name].unlink()
    assert build.outdated() == [str(files[name])]


def test_an_output_that_fails_to_build_leaves_the_old_one(tree, monkeypatch):
    build, files = tree
    old = files["host"].read_text()
    os.utime(files["host.cpp"], (3000, 3000))

    def command(out):
        return ["sh", "-c", f"echo half > {out}; exit 1"]
    monkeypatch.setattr(build, "_host_command", command)
    with pytest.raises(RuntimeError, match="host.cpp"):
        build.build()
    assert files["host"].read_text() == old and sorted(os.listdir(build.HERE)) == ["_host.so", "csrc", "lib.so"]
    monkeypatch.setattr(build, "_host_command", lambda out: ["sh", "-c", f"echo '[built for torch 1, Python x] new' > {out}"])
    build.build()
    assert files["host"].read_text().endswith("new\n") and not build.needs_build()


@pytest.mark.parametrize("other", ["torch 2, Python x", "torch 1, Python y"])
def test_a_host_module_for_another_torch_or_python_is_built_again(tree, monkeypatch, other):
    build, _ = tree
    monkeypatch.setattr(build, "built_for", lambda: other)
    assert build.outdated() == [build.HOST]


def test_the_host_module_says_what_it_was_built_for():
    import torch
    from lightop_b200 import _lib, build
    assert torch.__version__ in build.built_for() and _lib.host.built_for == f"[built for {build.built_for()}]"


@pytest.mark.parametrize("found", [False, True])
def test_the_library_needs_no_torch(tree, monkeypatch, tmp_path, found):
    # none installed, or one without CUDA
    build, files = tree
    spec = importlib.util.spec_from_file_location("torch", str(tmp_path / "__init__.py"), submodule_search_locations=[str(tmp_path)]) if found else None
    monkeypatch.setattr(importlib.util, "find_spec", lambda name: spec)
    monkeypatch.setattr(build, "host_possible", build.really_possible)
    files["host"].unlink()
    assert build.outdated() == []
    os.utime(files["a.cu"], (3000, 3000))
    assert build.outdated() == [build.LIB]


_IMPORT = """
import sys, types, warnings
import torch
case = sys.argv[1]
if case == "missing":
    sys.modules["lightop_b200._host"] = None          # (its import raises ImportError)
elif case == "other":
    sys.modules["lightop_b200._host"] = types.SimpleNamespace(built_for="[built for torch 1.0, Python x]")
elif case == "older":
    sys.modules["lightop_b200._host"] = types.SimpleNamespace()      # from before it said so
elif case == "cpu":
    sys.modules["lightop_b200._host"] = None
    torch.version.cuda = None
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    import lightop_b200 as lo
seen = [str(w.message) for w in seen if "_host.so" in str(w.message)]
assert len(seen) == (0 if case == "cpu" else 1) and all("build.py" in s for s in seen), seen
from lightop_b200 import _lib
assert _lib.load().lo_version() == 1
assert _lib.host.topk_softmax(1, 2, 3, 4) is None and _lib.host.fused_experts() is None and _lib.host.linear() is None
try:
    lo.moe.topk_softmax(torch.zeros(2, 2), torch.zeros(2, 2, dtype=torch.int32), None, torch.zeros(2, 8), True)
except RuntimeError as e:
    assert "CUDA" in str(e)
else:
    raise SystemExit("a CPU tensor was taken")
"""


@pytest.mark.parametrize("case", ["missing", "other", "older", "cpu"])
def test_the_package_works_without_the_host_module(case):
    subprocess.run([sys.executable, "-c", _IMPORT, case], cwd=ROOT, check=True, timeout=300)
