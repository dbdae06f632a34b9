"""The native artefact as a pair of libraries: the plain C one, and the operator binding that is compiled
against one torch.  What is kept or loaded for which torch, and what a failed or partial load leaves
behind.  Loads run in fresh interpreters; none touches CUDA."""
import json
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PRELUDE = r'''
import json, sys, warnings
sys.path.insert(0, sys.argv[1])
from __graft_entry__ import load_package
package = load_package()
import torch
from slidesparse_diffusion_b200 import backend
def native():
    """Is the forward path's CUDA kernel the compiled one?"""
    name = "sdacc_mild_projection_sm80::projection"
    return torch._C._dispatch_has_kernel_for_dispatch_key(name, "CUDA") and "ss_torch.cpp" in torch._C._dispatch_dump(name)
'''


def run(body, *arguments):
    done = subprocess.run([sys.executable, "-c", PRELUDE + body, str(ROOT), *map(str, arguments)], capture_output=True,
                          text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-3000:]
    return json.loads(done.stdout.strip().splitlines()[-1])


@pytest.fixture
def copy(backend, tmp_path):
    """A copy of the artefact, with changes to its receipt."""
    built = backend.default_directory()

    def make(files=(backend.LIBRARY_NAME, backend.BINDING_LIBRARY_NAME), name="native", **changes):
        target = tmp_path / name
        target.mkdir()
        for file in files:
            shutil.copy2(built / file, target / file)
        receipt = json.loads((built / "receipt.json").read_text())
        receipt.update(changes)
        (target / "receipt.json").write_text(json.dumps(receipt))
        return target
    return make


@pytest.mark.parametrize("changes", [dict(torch="0.0.0"), dict(cuda="0.0")])
def test_artefact_of_another_torch_is_built_again(backend, copy, monkeypatch, changes):
    target, built = copy(**changes), []

    def stop(command, **kwargs):
        built.append(command)
        raise RuntimeError("compiler called")

    monkeypatch.setattr(backend.subprocess, "run", stop)
    monkeypatch.setattr(backend.torch.cuda, "is_initialized", lambda: False)
    with pytest.raises(RuntimeError, match="compiler called"):
        backend.build_native(target)
    assert built
    assert backend.build_native(copy(name="same"))["complete"] and len(built) == 1        # an artefact of this torch is kept


@pytest.mark.parametrize("changes", [dict(torch="0.0.0"), dict(cuda="0.0")])
def test_binding_of_another_torch_is_not_loaded(copy, changes):
    """Its C++ types are another torch's; the C library beside it has none, and binds through ctypes."""
    result = run(r'''
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    package.load_native(sys.argv[2])
print(json.dumps(dict(native=native(), warned=[str(w.message) for w in seen if "rebuild" in str(w.message)])))
''', copy(**changes))
    assert not result["native"] and len(result["warned"]) == 1


def test_failed_load_leaves_nothing_behind(backend, copy):
    """A binding that cannot be loaded, twice, then a good directory in the same process."""
    broken = copy(name="broken")
    (broken / backend.BINDING_LIBRARY_NAME).write_bytes(b"not a library")
    receipt = json.loads((broken / "receipt.json").read_text())
    receipt["binding_sha"] = backend.sha(broken / backend.BINDING_LIBRARY_NAME)
    (broken / "receipt.json").write_text(json.dumps(receipt))
    result = run(r'''
errors = []
for _ in range(2):
    try:
        package.load_native(sys.argv[2])
        errors.append("")
    except OSError as error:
        errors.append(str(error))
package.load_native(sys.argv[3])
print(json.dumps(dict(errors=errors, native=native())))
''', broken, copy(name="good"))
    assert all(result["errors"]) and result["native"]


def test_names_taken_by_another_library_leave_nothing_behind():
    """The reference's own extension in the same process defines the same operator names."""
    result = run(r'''
other = torch.library.Library("sdacc_prepared_projection_sm80", "DEF")
errors = []
for _ in range(2):
    try:
        package.load_native()
        errors.append("")
    except RuntimeError as error:
        errors.append(str(error))
other.define("run(Tensor input,int handle,int n)->Tensor")
untouched = not torch._C._dispatch_has_kernel_for_dispatch_key("sdacc_prepared_projection_sm80::run", "CUDA")
other._destroy()
package.load_native()
print(json.dumps(dict(errors=errors, native=native(), untouched=untouched)))
''')
    assert all(result["errors"]) and result["native"] and result["untouched"]


def test_missing_binding_is_said_and_a_whole_copy_is_native(backend, copy):
    """The C library alone still binds every operator, but not without a word: its calls cost more host time."""
    body = r'''
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    package.load_native(sys.argv[2])
print(json.dumps(dict(native=native(), warned=[str(w.message) for w in seen if backend.BINDING_LIBRARY_NAME in str(w.message)],
                      defined=hasattr(torch.ops.slidesparse_b200, "projection_fused"))))
'''
    alone = run(body, copy((backend.LIBRARY_NAME,), name="alone"))
    assert not alone["native"] and alone["defined"] and len(alone["warned"]) == 1
    whole = run(body, copy(name="whole"))
    assert whole["native"] and whole["defined"] and not whole["warned"]
