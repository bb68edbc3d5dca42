"""The solver takes for granted how the trials of the face table are built (static assertions beside the kernels): a
table whose head-wave denominators are not the step's own length times the point's slowness does not compile."""
import os
import re
import subprocess

import pytest

from fdtomoc_gb300 import build as B

HEAD_1D = r"(\{FDN_1D,[^\n]*\{\{2,\{\{FDN_R,\{0,0,0\}\},\{FDN_DQ,\{0,0,0\}\}\}\}\},\{3,\{\{FDN_R,\{0,0,0\}\},\{)FDN_DQ(,\{0,0,0\}\},\{)FDN_SLOW"


@pytest.mark.parametrize("wrong", [None, r"\1FDN_DF\2FDN_SLOW", r"\1FDN_DQ\2FDN_S"])
def test_head_denominators_are_checked(tmp_path, wrong):
    table = open(os.path.join(B.CSRC, "fd_face_table.h")).read()
    if wrong:
        changed = re.sub(HEAD_1D, wrong, table, count=1)
        assert changed != table
        table = changed
    (tmp_path / "fd_face_table.h").write_text(table)
    for f in os.listdir(B.CSRC):   # beside the changed table, so that #include "..." finds it first
        if f.endswith((".h", ".cuh")) and f != "fd_face_table.h":
            (tmp_path / f).write_text(open(os.path.join(B.CSRC, f)).read())
    (tmp_path / "t.cu").write_text('#include <cuda_runtime.h>\n#include "fd_face_table.h"\n#include "fdgpu_layout.h"\n'
                                   '#include "fdgpu_check.cuh"\n#include "fdgpu_eval.cuh"\n#include "fdgpu_trials.cuh"\n')
    r = subprocess.run([B._nvcc()] + B.ARCH + B.NVFLAGS + ["-cuda", str(tmp_path / "t.cu"), "-o", str(tmp_path / "t.ii")],
                       capture_output=True, text=True)
    assert (r.returncode == 0) == (wrong is None), r.stderr
    assert wrong is None or "1-D trials" in r.stderr
