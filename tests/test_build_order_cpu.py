"""The order of importing the package, building its library and using it, in processes of their own with a copy of the
package's Python files and an empty extension module in the place of the linked library."""
import shutil
import subprocess
import sys
import sysconfig
import textwrap
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

STUB = """
#include <Python.h>
static PyObject* called(PyObject* self, PyObject* args) { return PyUnicode_FromString(LINK); }
static PyMethodDef calls[] = {FUNCTION {NULL, NULL, 0, NULL}};
static PyModuleDef def = {PyModuleDef_HEAD_INIT, "_C", NULL, -1, calls};
PyMODINIT_FUNC PyInit__C(void) { return PyModule_Create(&def); }
"""


def _link(target: Path, name: str, with_call: bool) -> None:
    """A library in a new file, as the linker leaves one."""
    src = target.parent / f"{name}.c"
    src.write_text(STUB)
    fresh = target.parent / f"{name}.so"
    function = '{"t_gemm", called, METH_VARARGS, NULL},' if with_call else ""
    subprocess.run(["gcc", "-shared", "-fPIC", f"-I{sysconfig.get_paths()['include']}", f'-DLINK="{name}"',
                    f"-DFUNCTION={function}", str(src), "-o", str(fresh)], check=True)
    fresh.replace(target)


@pytest.fixture
def tree(tmp_path):
    skip = shutil.ignore_patterns("_C*", "build", "csrc", "__pycache__")
    shutil.copytree(ROOT / "fluidmoe_b200", tmp_path / "fluidmoe_b200", ignore=skip)
    shutil.copy(ROOT / "__graft_entry__.py", tmp_path)
    shutil.copy(Path(__file__), tmp_path / "stub_link.py")
    return tmp_path


def _run(tree, body):
    head = """
        import sys
        import __graft_entry__ as entry
        from fluidmoe_b200 import _native, build
        from fluidmoe_b200.ops import gemm
        from stub_link import _link
        def linker(name):
            def run(verbose=True, force=False):
                _link(build.target_path(), name, True)
                return build.target_path()
            return run
    """
    script = textwrap.dedent(head) + textwrap.dedent(body)
    res = subprocess.run([sys.executable, "-c", script], cwd=tree, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr


@pytest.mark.parametrize("before", ["none", "older", "broken"])
def test_import_then_build_then_use(tree, before):
    """Importing loads nothing, so the first build of a process ends with the library that it has linked."""
    target = tree / "fluidmoe_b200" / ("_C" + sysconfig.get_config_var("EXT_SUFFIX"))
    if before == "older":
        _link(target, "old", False)
    elif before == "broken":
        target.write_bytes(b"no library")
    _run(tree, """
        assert "fluidmoe_b200._C" not in sys.modules
        build.build = linker("new")
        entry.build()
        assert _native.lib().__file__ == str(build.target_path()) and _native.is_current()
        assert gemm._t_gemm() == "new" and gemm._t_gemm is _native.lib().t_gemm
    """)


def test_failed_load_lasts_no_longer_than_its_file(tree):
    _run(tree, """
        def refused(call, word):
            try:
                call()
            except RuntimeError as e:
                assert word in str(e), e
            else:
                raise AssertionError(word)
        refused(_native.lib, "not built")
        refused(gemm._t_gemm, "not built")
        linker("new")()
        assert gemm._t_gemm() == "new"
        build.build = linker("newer")
        refused(entry.build, "new process")
    """)


def test_older_library_is_named_at_the_call(tree):
    _run(tree, """
        _link(build.target_path(), "old", False)
        try:
            gemm._t_gemm()
        except RuntimeError as e:
            assert "older than the package" in str(e)
        else:
            raise AssertionError
    """)
