"""The projector's copies into shared memory begin on their own size, at every
pitch of the volume's copy, and each of its forms adds a ray's terms in the
reference's order: a test program compiled from the library's own header runs it
beside the reference's plain loops on the same arithmetic (bits must agree)."""
import os
import subprocess

import pytest

from conftest import ROOT, geo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="session")
def program(tmp_path_factory):
    exe = tmp_path_factory.getbasetemp() / "projector_check"
    if exe.exists():  # built by another module's use of the fixture
        return str(exe)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "mcsart_b200", "csrc"),
                    "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "projector_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    return str(exe)


def run(program, cases):
    """cases: (geometry, pitch, angle).  Asserts that no copy is misaligned and no ray
    differs; returns each case's counts of the forms."""
    lines = [" ".join(repr(x) for x in (g["nx"], g["ny"], g["nz"], nzp, g["na"], g["nb"], g["SO"],
                                        g["SD"], g["da"], g["db"], g["ai"], g["bi"], angle))
             for g, nzp, angle in cases]
    out = subprocess.run([program], input="\n".join(lines) + "\n", capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr
    counts = [[int(x) for x in line.split()] for line in out.stdout.splitlines()]
    assert len(counts) == len(cases)
    for case, c in zip(lines, counts):
        assert c[:2] == [0, 0], (case, c)
    return [c[2:] for c in counts]


def test_copies_are_aligned_and_sums_are_the_plain_loops(program):
    """Narrow cells and cells wider than a voxel; a volume's copy has an odd pitch only
    where the even one does not fit (zf_pitch)."""
    cases = []
    for db in (0.8, 1.7):
        for nz, nzp in ((24, 24), (15, 16), (15, 15), (17, 17), (1, 1)):
            g = geo(nx=36, ny=32, nz=nz, na=21, nb=40, SO=90.0, SD=135.0, da=0.9, db=db, ai=0.3, bi=0.2)
            cases += [(g, nzp, angle) for angle in (0.3, 1.5)]
    run(program, cases)
