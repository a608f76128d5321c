"""What build() recompiles (CPU; the compilers are replaced by a recorder)."""
import os

import pytest

from fused_turboquant_b200 import build


@pytest.fixture
def outputs(tmp_path, monkeypatch):
    """Outputs that are up to date, in a folder of their own; the list of outputs build() makes."""
    made = []

    def fake_run(cmd, **kw):
        out = cmd[cmd.index("-o") + 1]
        made.append(out)
        with open(out, "wb") as f:
            f.write(" ".join(cmd).encode())
        return type("R", (), dict(returncode=0, stdout="", stderr=""))

    monkeypatch.setattr(build.subprocess, "run", fake_run)
    monkeypatch.setattr(build, "_nvcc", lambda: "/usr/local/cuda/bin/nvcc")
    monkeypatch.setattr(build, "OBJ_DIR", str(tmp_path / "build"))
    for name in ("LIB_PATH", "TEST_LIB_PATH", "NATIVE_PATH"):
        monkeypatch.setattr(build, name, str(tmp_path / (name + ".so")))
    build.build()
    made.clear()
    return made


def test_up_to_date_outputs_are_left_alone(outputs, monkeypatch):
    build.build()
    assert outputs == []
    # the host path is older than a kernel, which it does not include
    ages = {build.NATIVE_PATH: 150, build.LIB_PATH: 300, build.TEST_LIB_PATH: 300,
            os.path.join(build.CSRC, "ftq_attn_flow.cuh"): 200}
    monkeypatch.setattr(os.path, "getmtime", lambda p: ages.get(p, 100))
    build.build()
    assert outputs == []


def test_force_rebuilds_everything(outputs):
    build.build(force=True)
    text = " ".join(outputs)
    assert all(os.path.basename(p) in text for p in (build.LIB_PATH, build.TEST_LIB_PATH, build.NATIVE_PATH))


def test_another_torch_makes_the_host_path_stale(outputs, monkeypatch):
    import importlib.metadata
    real = importlib.metadata.version
    monkeypatch.setattr(importlib.metadata, "version", lambda n: "99.0" if n == "torch" else real(n))
    build.build()
    assert len(outputs) == 1 and os.path.basename(build.NATIVE_PATH) in outputs[0]
    build.build()
    assert len(outputs) == 1


def test_outputs_appear_complete(outputs):
    """Nothing is written under an output's own name: a process that has it loaded keeps its file."""
    build.build(force=True)
    assert not set(outputs) & {build.LIB_PATH, build.TEST_LIB_PATH, build.NATIVE_PATH}


@pytest.mark.parametrize("name", sorted(n for n in os.listdir(build.CSRC) if n.endswith(".cuh")))
def test_kernels_launched_early_do_not_load_through_the_read_only_path(name):
    """A kernel that waits for the one before it lives while that one writes: what it reads may not go through the cache
    that is not kept coherent (ftq_common.cuh: load8)."""
    with open(os.path.join(build.CSRC, name)) as f:
        code = "\n".join(line.split("//")[0] for line in f)
    if name != "ftq_common.cuh" and "after_previous_kernel()" in code:
        assert "__ldg" not in code and "ld.global.nc" not in code


@pytest.mark.parametrize("name", sorted(n for n in os.listdir(build.CSRC) if n.endswith(".cuh")))
def test_warps_are_whole_before_aligned_barriers(name):
    """`bar.sync` and `barrier.cluster ... .aligned` are undefined for a warp whose lanes arrive apart, and inline assembly
    does not bring them together: the statement before is a __syncwarp()."""
    with open(os.path.join(build.CSRC, name)) as f:
        code = [line.split("//")[0].strip() for line in f]
    code = [line for line in code if line]
    for before, line in zip(code, code[1:]):
        if "asm volatile(\"bar.sync" in line or ("barrier.cluster" in line and ".aligned" in line):
            assert before == "__syncwarp();", line


def test_a_wait_for_pages_has_one_answer_for_the_warp():
    """What follows it in the decode kernel (shuffles, MMAs, page requests) is run by all lanes or by none."""
    with open(os.path.join(build.CSRC, "ftq_attn_flow.cuh")) as f:
        waits = [line for line in f if "mbar_wait(my_bars" in line]
    assert waits and all("__all_sync(0xffffffffu, mbar_wait(" in line for line in waits)
