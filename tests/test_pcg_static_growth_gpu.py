"""psx_pcg_static reserves no device memory after its first call on a device, whatever the size
(cluster, grid and three-launch form), preconditioner and value type of later calls (GPU).

In a child process: what earlier tests have loaded would hide it."""
from __future__ import annotations

import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
    import ctypes, sys
    import numpy as np, torch
    sys.path[:0] = [{root!r}, {root!r} + "/tests"]
    from test_pcg_resident_gpu import _system
    from test_zz_no_alloc import _bind
    from psierra_b200 import _lib
    L = _bind()
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, dtype=d)).cuda()
    systems = []
    for n in (3000, 50001, 589998):
        A, b = _system(n, True, 1)
        systems.append((n, t(A.indptr, np.int32), t(A.indices, np.int32), (t(A.data, np.float64), t(A.data, np.float32)),
                        t(b, np.float64), torch.zeros(n, dtype=torch.float64, device="cuda")))
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    free = None
    for n, indptr, indices, values, b, x in systems:
        for precond in (_lib.PSX_PRECOND_JACOBI, _lib.PSX_PRECOND_NONE, _lib.PSX_PRECOND_BJACOBI,
                        _lib.PSX_PRECOND_BJACOBI | _lib.PSX_PCG_NODAL, _lib.PSX_PRECOND_JACOBI | _lib.PSX_PCG_NODAL):
            for vp, v in zip((_lib.PSX_FP64, _lib.PSX_FP32_MIXED), values):
                x.zero_()
                torch.cuda.synchronize()
                rc = L.psx_pcg_static(n, indptr.data_ptr(), indices.data_ptr(), v.data_ptr(), vp, b.data_ptr(), x.data_ptr(),
                                      1e-8, 0.0, 500, precond, status.data_ptr(), torch.cuda.current_stream().cuda_stream)
                torch.cuda.synchronize()
                now = torch.cuda.mem_get_info()[0]
                assert rc == 0 and status.tolist()[5] == 0
                assert free is None or now == free, (n, precond, vp, free - now)
                free = now
"""


def test_later_calls_of_other_sizes_and_options_reserve_nothing():
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(CHILD).format(root=ROOT)], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
