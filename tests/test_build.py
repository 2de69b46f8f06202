"""CPU tests of the build rules: the C libraries and the harness need nvcc only, and the torch binding is built anew for
another torch or interpreter; and of one rule of the sources that no run can show."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hopper_jeni_b200", "csrc")


def _dry_run(*args):
    return subprocess.run(["make", "-n", "-C", CSRC, *args], capture_output=True, text=True)


def test_default_target_needs_no_python_and_no_torch():
    out = _dry_run("-B", "PYTHON=/nonexistent", "CXX=/nonexistent")
    assert out.returncode == 0, out.stderr
    assert "libgqa_b200.so" in out.stdout
    assert "_gqa_torch" not in out.stdout and "/nonexistent" not in out.stdout + out.stderr


def test_binding_is_rebuilt_for_another_abi():
    assert "torch_binding.cpp" not in _dry_run("binding").stdout  # built, up to date
    assert "torch_binding.cpp" in _dry_run("binding", "BINDING_ABI=another-torch-or-interpreter").stdout


def test_forward_takes_tensor_memory_behind_its_wait():
    """The forward may come up under the end of any kernel, also of one that has let it start before taking its own tensor
    memory: holding some while it waits for that kernel's end, it could keep it from ever ending."""
    with open(os.path.join(CSRC, "gqa_fwd_sm100.cu")) as f:
        src = f.read()
    assert 0 < src.rindex("pdl_wait();") < src.index("tmem_alloc(")
