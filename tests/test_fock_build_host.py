"""Host side of vlxb_fockBuild against fakes of the list preparations and the
kernel launchers (fock_build_host.cu); no GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = os.environ.get("NVCC", "nvcc")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    if not shutil.which(NVCC):
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("fockbuild") / "harness")
    subprocess.run([NVCC, "-std=c++17", "-O0", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                    os.path.join(HERE, "fock_build_host.cu")], check=True, capture_output=True, text=True)

    def run(scenario, number=0):
        r = subprocess.run([exe, scenario, str(number)], check=True, capture_output=True, text=True, timeout=60)
        return {k: int(v) for k, v in (ln.split() for ln in r.stdout.splitlines())}

    return run


@pytest.mark.parametrize("scenario", ["cutoff set", "cutoff reset", "budget set"])
@pytest.mark.parametrize("reads", [1, 2, 3, 4, 5, 6, 8])
def test_fp32_settings_are_read_once_per_build(harness, scenario, reads):
    """Settings that another thread changes during a build (after `reads` reads):
    every preparation and every launch goes by one value of each.  A launch with
    a cutoff on lists prepared without one has no partner groups to read."""
    r = harness(scenario, reads)
    assert r["rc"] == 0 and r["launches"] in (2, 4), r  # one pass per kind, or two
    assert r["null_groups"] == r["null_sums"] == r["cut_differs"] == 0, r


@pytest.mark.parametrize("number", [0, 1, 2, 3])
def test_memory_runs_out_before_or_after_the_first_launch(harness, number):
    """VLXB_ENOMEM (3) tells the caller that no output was touched and that the
    class calls may go on: so it comes from a preparation.  An allocation error
    of a launch (of a kernel's first load, say) is VLXB_ECUDA (2), as other
    classes have added to the outputs by then."""
    r = harness("preparation fails", min(number, 2))  # three record lists, four launches
    assert r["launches"] == 0 and r["rc"] == 3, r
    r = harness("launch fails", number)
    assert r["launches"] == number + 1 and r["rc"] == 2, r


@pytest.mark.parametrize("missing,rc", [
    (0, 0), (1, 1), (2, 1), (4, 1),
    (8, 0), (8 + 1, 1), (8 + 2, 1), (8 + 4, 0),  # Coulomb class alone: molecules of p and d primitives
    (16 + 2, 0), (16 + 8 + 3, 0),                # an empty Coulomb list needs none
])
def test_batch_without_molecules_is_refused(harness, missing, rc):
    """A batch (n_mol > 0) whose Coulomb classes have no molecule of their
    primitives is refused as by vlxb_coulombBatch, before anything is queued:
    without them every molecule would meet the kets of all others."""
    r = harness("batch", missing)
    assert r["rc"] == rc, r
    assert rc == 0 or r["prepared"] == r["launches"] == 0, r


def test_density_columns_and_stride_belong_to_a_batch(harness):
    """prim_aocols and D_stride are read for n_mol > 0 alone (vlxb.h): one
    molecule's density has the rows' indices and naos columns."""
    r = harness("columns", 0)
    assert (r["rc"], r["col_index"], r["stride"]) == (0, 0, 5), r
    r = harness("columns", 2)
    assert (r["rc"], r["col_index"], r["stride"]) == (0, 8, 3), r
