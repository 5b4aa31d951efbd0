"""A product behind a caller's kernel that runs for longer than the GEMMs' bounded waits (about 2 s) after
letting the product's first kernel start: the limits of the waits count from that kernel's end."""
import ctypes
import os
import subprocess
import time

import numpy as np
import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def early_release(tmp_path_factory):
    out = tmp_path_factory.mktemp("early_release") / "early_release.so"
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-shared", "-Xcompiler", "-fPIC",
                    os.path.join(REPO, "tests", "native", "early_release.cu"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    lib.early_release.argtypes = [ctypes.c_ulonglong, ctypes.c_uint, ctypes.c_void_p]
    return lib.early_release


@pytest.mark.parametrize("limbs", [28, 60])
def test_product_behind_a_long_kernel_that_released_it(limbs, early_release, fpc, inputs, oracle):
    import torch
    n = 4096
    q, a, b = inputs.instance(n, limbs, 12, 0)
    with fpc.Plan(n, 32 * limbs, limbs, q) as plan:
        da, db = (torch.from_numpy(x.view(np.int32)).cuda() for x in (a, b))
        dc = torch.full_like(da, -1)
        stream = torch.cuda.current_stream().cuda_stream
        call = lambda: plan.run_device(da.data_ptr(), db.data_ptr(), dc.data_ptr(), stream)  # noqa: E731
        call()
        assert early_release(0, 1, stream) == 0
        torch.cuda.synchronize()
        dc.fill_(-1)
        torch.cuda.synchronize()
        start = time.perf_counter()
        assert early_release(3_000_000_000, 4_000_000, stream) == 0
        call()
        torch.cuda.synchronize()
        assert time.perf_counter() - start > 2.5
        assert plan.status() == 0
        assert np.array_equal(dc.cpu().numpy().view(np.uint32), oracle.kronecker(q, a, b))
