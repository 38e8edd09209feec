"""How many planes a block of the field passes marches and how many slices a
block of the denoiser's convolutions streams is chosen from the grid. The sizes
at which the GPU tests compare those kernels with the oracle have to reach the
march and the stream, a last block with fewer planes among them: the rules
themselves, compiled for the host, say so."""
import os
import shutil
import subprocess

import pytest

from test_gpu_denoiser import SLICES
from test_gpu_field_layers import MARCHED

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("rules") / "block_rules_harness")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(HERE, "..", "rhybrid_b200", "csrc"), "-o", exe,
                    os.path.join(HERE, "block_rules_harness.cu")], check=True)

    def of(sizes):
        text = "".join("%d %d %d\n" % s for s in sizes)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]

    return of


def test_marched_planes(rules):
    got = rules([d for d, _, _ in MARCHED])
    for (dims, node, cell), (n, c, _) in zip(MARCHED, got):
        assert (n, c) == (node, cell), dims
    assert {2, 4, 8} <= {n for _, n, _ in MARCHED} and {2, 4, 8} <= {c for _, _, c in MARCHED}
    assert all(d[2] % max(n, c) for d, n, c in MARCHED)


def test_streamed_slices(rules):
    got = rules([d for d, _ in SLICES])
    for (dims, zc), (_, _, z) in zip(SLICES, got):
        assert z == zc and dims[2] % zc, dims


def test_full_size_grids_march_and_stream(rules):
    (node, cell, slices), = rules([(120, 160, 160)])
    assert (node, cell, slices) == (8, 8, 12)


def test_long_axes_fit_the_launch(rules):
    """At most 65535 blocks along z for every nz that eight slices per block fit."""
    sizes = [(3, 3, nz) for nz in range(65536, 8 * 65535 + 1, 1013)] + [(3, 3, 8 * 65535)]
    for (_, _, nz), (_, _, z) in zip(sizes, rules(sizes)):
        assert (nz + z - 1) // z <= 65535, nz
