"""Index arithmetic of kernels that run a warp per row, at row counts whose
threads no longer fit in 32 bits (2^27 rows and more); on the host."""
import pathlib
import subprocess

from test_device_functors import _nvcc

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_warp_per_row_beyond_2_27_rows(tmp_path):
    exe = tmp_path / "warp_index_check"
    subprocess.check_call([_nvcc(), "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                           str(ROOT / "race_gb300" / "csrc"), "-I", str(ROOT / "include"),
                           str(ROOT / "tests" / "warp_index_check.cu"), "-o", str(exe)])
    rows = [1, 7, 8, 9, 2 ** 27 - 1, 2 ** 27, 2 ** 27 + 1, 513 ** 3, 2 ** 28 + 5, 2 ** 31 - 1]
    got = subprocess.run([str(exe), *map(str, rows)], capture_output=True, text=True)
    assert got.stdout == "" and got.returncode == 0, "rows run by another warp: " + got.stdout.replace("\n", " ")
