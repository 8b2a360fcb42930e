"""The batched solver's rate tables in shared memory and, above 32 KB, in the workspace (gpu), in one process:
against the oracle's solve within Expokit's budget, and one table per cluster beside the basis, not one per CTA."""
import re

import numpy as np
import pytest

import oracle
from cuda_fsp_b200 import BatchKrylov, models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 128), (8, 256), (16, 512)])
def test_both_places(cuda, shape):
    t, tol = 30.0, 1e-9
    for box in [(700, 3), (30, 21), (2, 900)]:  # 39 KB, 3 KB and 51 KB of tables
        ms = [models.toggle((box[0] - k % 2, box[1] + k % 3)) for k in range(6)]
        B = BatchKrylov.from_models(ms, m=20, tol=tol)
        B.set_shape(*shape)
        p = B.pack([mm.p0() for mm in ms])
        for _ in range(2):  # the tables are written anew for each instance and solve
            p.copy_(B.pack([mm.p0() for mm in ms]))
            stats = B.solve(t, p)
        for mm, w, st in zip(ms, B.unpack(p), stats):
            ref, _, rc = oracle.expv(oracle.assemble_model(mm), mm.coefs(0.0), t, mm.p0(), m=20, tol=tol)
            assert rc == 0 and st["status"] == 0
            assert np.abs(w - ref).sum() <= 2.4 * tol * t


def test_workspace_of_a_long_axis(cuda):
    import torch
    ms = [models.toggle((400000, 1)) for _ in range(8)]
    B = BatchKrylov.from_models(ms, m=10, tol=1e-8)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    B.set_shape(16, 512)
    used = free - torch.cuda.mem_get_info()[0]
    clusters = int(re.search(r"(\d+) clusters", B.describe()).group(1))
    n, stride, nr = ms[0].n_states, 400003, ms[0].nr
    assert used <= 8 * clusters * (11 * n + (nr + 1) * stride) + (32 << 20)  # kernels and page rounding: 32 MB


def test_solve_after_a_shape_without_workspace(cuda):
    """set_shape that finds no memory gives the workspace of the earlier shape back: the next solve must not use
    it, and chooses a shape that fits."""
    import torch
    from cuda_fsp_b200 import CufspError
    ms = [models.toggle((699, 699)) for _ in range(40)]
    B = BatchKrylov.from_models(ms, m=30, tol=1e-8)
    B.set_shape(16, 512)
    p0 = B.pack([mm.p0() for mm in ms])
    p, q = p0.clone(), p0.clone()
    B.solve(1e-3, p)
    per_cluster = 8 * 31 * ms[0].n_states  # 122 MB
    wide = int(re.search(r"(\d+) clusters", B.describe()).group(1))
    torch.cuda.synchronize()
    filler = torch.empty((torch.cuda.mem_get_info()[0] - 2 * per_cluster) // 8, dtype=torch.float64, device="cuda")
    with pytest.raises(CufspError) as e:
        B.set_shape(2, 128)  # more clusters than `wide` + 2
    assert e.value.name == "CUFSP_ERR_ALLOC"
    del filler
    torch.cuda.empty_cache()
    B.solve(1e-3, q)
    assert int(re.search(r"(\d+) clusters", B.describe()).group(1)) >= 1 and wide + 2 < 40
    assert (p - q).abs().sum().item() <= 1e-9
