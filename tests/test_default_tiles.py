"""default_ops (csrc/registry.cu): which tile a mesh takes without tuning."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
MIXED = 1000
EULER2D, EULER3D, NS3D = 1, 8, 9
SECOND_FORM = 3

# (key, p, elements per SM, and one more, boundary sides) -> (kind or None, threads or None)
CASES = [((EULER3D, p, 40, 0, 0), (SECOND_FORM, None)) for p in (2, 3, 4)]
CASES += [((EULER3D + MIXED, p, 40, 0, 0), (SECOND_FORM, None)) for p in (2, 3, 4)]
CASES += [((EULER3D, p, n, 0, 1), (0, None)) for p in range(1, 8) for n in (1, 40)]     # walls
CASES += [((EULER3D + MIXED, p, 1, k, 0), (0, 256 if k else 512)) for p in (6, 7) for k in (0, 1)]
CASES += [((NS3D, p, 5, k, 0), (0, 64 if k else 128)) for p in (1, 2) for k in (0, 1)]
CASES += [((NS3D, 3, 14, k, 0), (0, 96 if k else 128)) for k in (0, 1)]
CASES += [((EULER2D, 5, 40, 0, 0), (0, 64)), ((EULER2D, 6, 28, 0, 0), (0, 64)), ((EULER2D, 6, 28, 1, 0), (0, 128)),
          ((EULER2D, 6, 16, 0, 0), (0, 128)), ((EULER2D, 6, 4, 0, 0), (0, 256))]


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    import dgm_b200
    lib = dgm_b200.lib()._name
    exe = str(tmp_path_factory.mktemp("tiles") / "tile_defaults")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(cuda, "include"), os.path.join(HERE, "tile_defaults.cpp"),
                    "-o", exe, lib, "-Wl,-rpath," + os.path.dirname(lib), "-L", os.path.join(cuda, "lib64"), "-lcudart"],
                   check=True, capture_output=True, text=True)
    args = [str(v) for a, _ in CASES for v in a]
    out = subprocess.run([exe] + args, check=True, capture_output=True, text=True).stdout.split("\n")
    return [tuple(int(v) for v in line.split()) for line in out[1:] if line]


@pytest.mark.parametrize("i", range(len(CASES)))
def test_default_tile(rows, i):
    (kind, threads), got = CASES[i][1], rows[i]
    assert got[0] == kind and threads in (None, got[1]), (CASES[i][0], got)
