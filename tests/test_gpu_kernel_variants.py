"""GPU: internal launches compared with one another or with values formed on the host
(tests/cpp/kernel_variants.cu, compiled against the in-tree library)."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def variants(handle, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no CUDA compiler")
    exe = tmp_path_factory.mktemp("variants") / "kernel_variants"
    lib_dir = ROOT / "quantkos_b200"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++20", "--expt-relaxed-constexpr",
                    f"-I{ROOT / 'include'}", f"-I{lib_dir / 'csrc'}", str(ROOT / "tests" / "cpp" / "kernel_variants.cu"),
                    f"-L{lib_dir}", "-lquantkos_b200", f"-Xlinker=-rpath,{lib_dir}", "-o", str(exe)],
                   check=True, capture_output=True, text=True)

    def run(section: str, at_least: int) -> None:
        r = subprocess.run([str(exe), section], capture_output=True, text=True, timeout=300)
        lines = r.stdout.splitlines()
        assert r.returncode == 0 and not [ln for ln in lines if ln.startswith("FAIL")], r.stdout + r.stderr
        assert len([ln for ln in lines if ln.startswith("ok ")]) >= at_least

    return run


def test_select_equals_sort(variants):
    """Ranks next to one another, ties, neighbouring bit patterns, subnormals and infinities, at
    sizes around a block and with several values per thread: bit for bit."""
    variants("select", 36)


def test_price_beside_a_distribution(variants):
    """A one-leg contract's price from its stored payoffs has the bits of the price alone; a
    contract of several legs is not priced from one leg's payoffs."""
    variants("distribution", 20)


def test_launch_shapes_give_the_same_records(variants):
    """Tile records of one task, bit for bit: one warp per tile, persistent blocks of 128, 256 and
    512 threads in one block and in 37, and with the term table."""
    variants("shapes", 65)


def test_slabs_with_and_without_a_term_table(variants):
    """400,003 paths of both models, bit for bit: two paths per thread with the table and without,
    one path per thread."""
    variants("slabs", 13)


def test_fp64_functions_against_long_double(variants):
    """The path kernels' own logarithm, exponential, reciprocal, roots and Box-Muller: a million
    arguments each, the edges of the words and of the tables, next to 1, out of range."""
    variants("functions", 11)
