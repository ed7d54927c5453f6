"""bench.py's roofline takes the path of the contractions from the library, not from their speed."""
import bench


class _Problem:
    npix, nuv, npow, nbis, width = 256 * 256, 21120, 21120, 70400, 256

    def dft_flops(self):
        return 4.0 * self.npix * self.nuv + 8.0 * self.width * self.nuv


def _measured(ms, uv_grid):
    stages = ("prep", "forward_dft", "vis_data", "adj_weights", "adjoint_dft", "grad_finalize")
    return {"stage_ms": {k: ms if k == "forward_dft" else 0.1 * ms for k in stages}, "stage_n": {k: 1 for k in stages},
            "uv_grid": uv_grid}


def test_bound_follows_the_path():
    p = _Problem()
    # 5.5 GFLOP of direct sums: 25 us would be 220 TFLOP/s (660 with three products), 1 us more than the tensor cores have
    for ms in (0.025, 0.001):
        for precision in ("fp32", "split16", "split16f8"):
            grid = bench.roofline(p, _measured(ms, True), precision, "precision")
            assert grid["bound"] == "hbm" and grid["uv_grid"] and "executed_tflops" not in grid and grid["traffic"] is None
            assert grid["work_per_launch"] == bench._grid_bytes(p)
            direct = bench.roofline(p, _measured(ms, False), precision, "precision")
            assert direct["bound"] == "tensor" and not direct["uv_grid"]
            assert direct["work_per_launch"] == p.dft_flops() and direct["executed_tflops"] >= direct["achieved"]


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    """Where the reference's sources were never there to compile, its arm says so in its line."""
    import argparse
    import json

    def missing(*_):
        raise FileNotFoundError("libgpair_ref.so not built (reference sources unavailable)")

    monkeypatch.setattr(bench, "reference_sample", missing)
    bench.run_reference(argparse.Namespace(workload="tiny", gpus=1, steps=1, warmup=3), 0)
    lines = capsys.readouterr().out.strip().splitlines()
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert line["impl"] == "reference" and "not built" in line["unavailable"] and len(line) == 2
