"""The in-tree build against a stand-in for nvcc (no CUDA): what is rebuilt, what a failure leaves, two builds at once."""
import os
import subprocess
import sys
import time

import pytest

from kerrsplat_b200 import build as b

NVCC = """#!{python}
import os, sys, time
a = sys.argv[1:]
out = a[a.index("-o") + 1]
with open("{log}", "a") as f:
    f.write(os.path.basename(out) + "\\n")
if "-c" in a:
    src = a[a.index("-c") + 1]
    text = open(src).read()
    with open(out, "w") as f:
        f.write("half")
        f.flush()
        time.sleep(30 if "slow" in text else 0.2)
        f.write(" fast " if "--use_fast_math" in a else " exact ")
        f.write(text)
    sys.exit(1 if "bad" in text else 0)
with open(out, "w") as f:
    f.write("|".join(open(o).read() for o in a if o.endswith(".o")))
"""


@pytest.fixture
def tree(tmp_path, monkeypatch):
    pkg = tmp_path / "pkg"
    (pkg / "csrc").mkdir(parents=True)
    (tmp_path / "include").mkdir()
    (tmp_path / "include" / "kerrsplat_b200.h").write_text("")
    for name in ("a.cu", "b.cu", "h.cuh"):
        (pkg / "csrc" / name).write_text(name)
    past = time.time() - 100
    for p in list((pkg / "csrc").iterdir()) + [tmp_path / "include" / "kerrsplat_b200.h"]:
        os.utime(p, (past, past))
    nvcc = tmp_path / "nvcc"
    nvcc.write_text(NVCC.format(python=sys.executable, log=tmp_path / "log"))
    nvcc.chmod(0o755)
    monkeypatch.setenv("NVCC", str(nvcc))
    monkeypatch.delenv("KS_FAST_MATH", raising=False)
    for k, v in dict(HERE=str(pkg), CSRC=str(pkg / "csrc"), LIB=str(pkg / "lib.so"), OBJECTS=str(pkg / "_build"), SOURCES=["a.cu", "b.cu"],
                     HEADERS=["h.cuh"]).items():
        monkeypatch.setattr(b, k, v)
    return tmp_path


def calls(tree):
    log = (tree / "log").read_text().split() if (tree / "log").exists() else []
    (tree / "log").write_text("")
    return sorted(log)


def test_flags_and_edits_decide_what_is_rebuilt(tree, monkeypatch):
    lib = tree / "pkg" / "lib.so"
    b.build(verbose=False)
    exact = lib.read_text()
    assert exact == "half exact a.cu|half exact b.cu" and calls(tree) == ["a.o.tmp", "b.o.tmp", "lib.so.tmp"]
    b.build(verbose=False)
    assert calls(tree) == []
    monkeypatch.setenv("KS_FAST_MATH", "1")
    b.build(verbose=False)
    assert lib.read_text() == exact.replace("exact", "fast") and calls(tree) == ["a.o.tmp", "b.o.tmp", "lib.so.tmp"]
    monkeypatch.delenv("KS_FAST_MATH")
    b.build(verbose=False)   # the objects of the other flags are still there, the library is not
    assert lib.read_text() == exact and calls(tree) == ["lib.so.tmp"]
    (tree / "pkg" / "csrc" / "b.cu").write_text("edited")
    b.build(verbose=False)
    assert lib.read_text() == "half exact a.cu|half exact edited" and calls(tree) == ["b.o.tmp", "lib.so.tmp"]


def test_a_failed_compile_leaves_the_library_and_stops_the_others(tree):
    b.build(verbose=False)
    before = (tree / "pkg" / "lib.so").read_text()
    (tree / "pkg" / "csrc" / "a.cu").write_text("bad")
    (tree / "pkg" / "csrc" / "b.cu").write_text("slow")
    t = time.time()
    with pytest.raises(subprocess.CalledProcessError):
        b.build(verbose=False)
    assert time.time() - t < 15
    assert (tree / "pkg" / "lib.so").read_text() == before
    assert not list((tree / "pkg").rglob("*.tmp")) and b.stale()


def test_two_builds_at_once(tree):
    code = "from kerrsplat_b200 import build as b\n" + "".join(
        f"b.{k} = {getattr(b, k)!r}\n" for k in ("HERE", "CSRC", "LIB", "OBJECTS", "SOURCES", "HEADERS")) + "b.build(verbose=False)\nprint(open(b.LIB).read())"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    two = [subprocess.Popen([sys.executable, "-c", code], cwd=root, stdout=subprocess.PIPE, text=True) for _ in range(2)]
    assert [p.communicate(timeout=60)[0].strip() for p in two] == ["half exact a.cu|half exact b.cu"] * 2
    assert calls(tree) == ["a.o.tmp", "b.o.tmp", "lib.so.tmp"]
