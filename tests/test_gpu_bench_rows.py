"""The bench's kernel rows name what runs: one row for a forward pass that also solves,
two where the plan's inversion keeps the solve apart (one tall field; the CUDA-core
engine), and a derived time is marked as such."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


@pytest.mark.parametrize("ny,nx,B,engine,rows", [
    (128, 128, 2, 0, {"dst-fwd-solve": "dst_tc_fwd_kernel"}),
    (1100, 90, 1, 0, {"dst-fwd": "dst_tc_fwd_kernel", "tridiag": "tridiag_chunked_kernel"}),
    (128, 128, 2, 1, {"dst-fwd": "dst_gemm_kernel", "tridiag": "tridiag_chunked_kernel"})])
def test_forward_rows(ny, nx, B, engine, rows):
    import bench
    from vardyn_gb300.qg1l import QG1LPlan
    p = QG1LPlan(ny, nx, 5e3, 5e3, 900.0, 1e-4, 2.7, dtype=torch.float32)
    p.set_schedule(engine=engine)
    table = {r["name"]: r for r in bench.kernel_table(p, B, 1, reps=20)}
    got = {k: r["kernel"].split("<")[0] for k, r in table.items() if k in ("dst-fwd", "tridiag", "dst-fwd-solve")}
    assert got == rows
    for k in rows:
        assert table[k]["algorithmic_bytes"] == 2 * B * ny * nx * 4
    if "dst-fwd-solve" in rows:
        r = table["dst-fwd-solve"]
        assert r["derived"] and (r["us"] is None) == (r["gbs"] is None)
    line, kernels, _ = bench.roofline_from_table(list(table.values()), 1.0, B, ny, {})
    assert line["kernel"] in [k["kernel"] for k in kernels]
