"""A kernel that could not be launched must end its call with an error: the node-side pass would otherwise add up
old partial sums and the call return success.  The functions that enqueue an apply return the launch's status,
and the build refuses code that drops it."""
import os
import shutil
import subprocess

import pytest

from immersed_catmull_clark_b200 import build as B

CALLS = {
    "contract": "o.enqueue_contract(nullptr, nullptr, nullptr)",
    "apply": "o.enqueue_apply(nullptr, nullptr, nullptr, nullptr)",
    "apply_on": "o.enqueue_apply_on(nullptr, nullptr, nullptr)",
    "pcg_iteration": "o.enqueue_pcg_iteration()",
    "pcg_modal": "o.enqueue_pcg_modal(1)",
    "modal_apply": "launch_modal_apply<double>(nullptr, m, s, t)",
    "modal_pcg": "launch_modal_pcg<double>(nullptr, m, s, t, 1, nullptr, 1)",
}


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
@pytest.mark.parametrize("call", sorted(CALLS))
def test_a_dropped_launch_status_does_not_compile(call, tmp_path):
    def compiles(statement):
        src = tmp_path / "probe.cu"
        src.write_text('#include <vector>\n#include "icc_device.cuh"\n#include "icc_modal.cuh"\n'
                       "namespace icc {\nbool probe(Op &o, const ModalHost &m, const ModalSys<double> &s, const ModalTile &t) {\n"
                       "    (void)o, (void)m, (void)s, (void)t;\n    " + statement + "\n}\n}\n")
        flags = [f for f in B.NVCC_FLAGS if f != "-shared"]
        r = subprocess.run(["nvcc", *flags, "-I", B.CSRC, "-c", str(src), "-o", os.devnull], capture_output=True, text=True)
        return r.returncode == 0, r.stderr

    ok, err = compiles(f"return {CALLS[call]} == cudaSuccess;")
    assert ok, err
    ok, err = compiles(f"{CALLS[call]}; return true;")
    assert not ok and "nodiscard" in err
