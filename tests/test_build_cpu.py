"""Building and importing: several processes at once, and a tree that was never built."""

import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

BUILDER = """
import sys, time
from pathlib import Path
from vllm_rlt_b200 import _build

_build.PACKAGE = Path(sys.argv[1])

def compiler(cmd, show=False):  # takes its time, and has written half of its output for most of it
    out = Path(cmd[cmd.index("-o") + 1])
    with open(_build.PACKAGE / "log", "a") as log:
        log.write("ran\\n")
    out.write_bytes(b"half")
    time.sleep(1.0)
    out.write_bytes(b"half and half")

_build._run = compiler
while not (_build.PACKAGE / "go").exists():
    time.sleep(0.001)
target = _build.build_library()
assert target.read_bytes() == b"half and half", target.read_bytes()
_build.build_library()
"""


def test_processes_that_start_together_build_once_and_never_see_half_a_library(tmp_path):
    workers = [subprocess.Popen([sys.executable, "-c", BUILDER, str(tmp_path)], cwd=ROOT, stderr=subprocess.PIPE) for _ in range(4)]
    (tmp_path / "go").touch()
    for worker in workers:
        _, err = worker.communicate(timeout=120)
        assert worker.returncode == 0, err.decode()[-2000:]
    assert (tmp_path / "log").read_text() == "ran\n"
    assert sorted(p.name for p in tmp_path.iterdir() if p.name[0] != ".") == ["go", "librlt_kv_handoff.so", "librlt_kv_handoff.so.stamp", "log"]


def test_importing_the_worker_modules_loads_and_builds_nothing(tmp_path):
    code = (
        "import sys\n"
        "from pathlib import Path\n"
        "from vllm_rlt_b200 import _build, _lib\n"
        f"_lib.HOST_PATH = _lib.LIB_PATH = Path({str(tmp_path)!r}) / 'missing.so'\n"
        "def build(*args, **kw): raise RuntimeError('a build')\n"
        "_build.build_library = _build.build_host = build\n"
        "from vllm_rlt_b200.worker import staging, tensors\n"
        "for use in (lambda: tensors.TensorTransfer, lambda: staging.StagedInputTensor, lambda: staging.StagedWriteTensor):\n"
        "    try:\n"
        "        use()\n"
        "    except RuntimeError as e:\n"
        "        assert str(e) == 'a build'\n"
        "    else:\n"
        "        raise AssertionError('a class without its base')\n"
    )
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=ROOT, timeout=120)
    assert done.returncode == 0, done.stderr[-2000:]


def test_the_classes_made_on_demand_are_the_same_every_time():
    from vllm_rlt_b200.worker import staging, tensors

    assert staging.TensorTransfer is tensors.TensorTransfer
    for module, name in ((tensors, "TensorTransfer"), (staging, "StagedInputTensor"), (staging, "StagedWriteTensor")):
        made = getattr(module, name)
        assert made is getattr(module, name) and made.__name__ == made.__qualname__ == name and made.__module__ == module.__name__
        assert made.__doc__
