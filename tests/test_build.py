"""CPU: when the host path's module is rebuilt, and that processes starting together build it once."""
import os
import subprocess
import sys
import textwrap

import pytest

from hdla_impl_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_built_module_says_what_it_was_built_for():
    assert build.binding_built_for(build.build_binding()) == build._torch_version()


@pytest.mark.parametrize("content,age,stale", [
    (None, 0, True), ("this", 0, False), ("this", -1e6, True), ("other", 0, True), ("", 0, True)])
def test_staleness(tmp_path, monkeypatch, content, age, stale):
    """Missing, older than its source, built for another PyTorch, or not saying: to be built again."""
    so = tmp_path / "_binding.so"
    monkeypatch.setattr(build, "BINDING", str(so))
    if content is not None:
        version = {"this": build._torch_version(), "other": "1.0.0", "": ""}[content]
        so.write_bytes(b"\x7fELF..." + (build._BUILT_FOR + version).encode() + b"\0rest" if version else b"\x7fELF")
        t = max(os.path.getmtime(f) for f in build._binding_sources()) + 10 + age
        os.utime(so, (t, t))
    assert build._binding_stale() == stale


def test_processes_that_start_together_build_once_and_find_a_whole_file(tmp_path):
    """Three processes without the module; the compiler is a stand-in that writes its output slowly, in two pieces."""
    log = tmp_path / "log"
    gxx = tmp_path / "g++"
    gxx.write_text(textwrap.dedent(f"""\
        #!{sys.executable}
        import sys, time
        open({str(log)!r}, "a").write("start\\n")
        marker = [a for a in sys.argv if a.startswith("-DHDLA_BUILT_FOR=")][0].split("=", 1)[1].strip('"')
        with open(sys.argv[sys.argv.index("-o") + 1], "wb") as f:
            f.write(b"first half, "); f.flush(); time.sleep(1.0)
            f.write(marker.encode() + b"\\0second half")
        open({str(log)!r}, "a").write("end\\n")
        """))
    gxx.chmod(0o755)
    so = tmp_path / "_binding.so"
    code = textwrap.dedent(f"""\
        from hdla_impl_b200 import build
        build.BINDING = {str(so)!r}
        assert open(build.build_binding(), "rb").read().endswith(b"second half")
        """)
    env = dict(os.environ, PATH=f"{tmp_path}{os.pathsep}{os.environ['PATH']}", PYTHONPATH=ROOT)
    procs = [subprocess.Popen([sys.executable, "-c", code], env=env) for _ in range(3)]
    assert [p.wait(timeout=120) for p in procs] == [0, 0, 0]
    assert log.read_text().split() == ["start", "end"]
    assert {p.name for p in tmp_path.iterdir()} == {"log", "g++", "_binding.so", "_binding.so.lock"}
