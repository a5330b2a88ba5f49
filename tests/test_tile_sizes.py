"""The tile sizes that the switches of the expert kernels choose among: a size that no kernel has would outgrow the tile list's
scratch or a kernel's stages, so whatever is asked for selects one that exists (compiled for the host, no GPU)."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "strata_b200", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    path = tmp_path_factory.mktemp("tiles") / "tiles.so"
    code = f'''#include "{CSRC}/tile_sizes.h"
extern "C" int plane_tile(int asked) {{ return smoe::existing_tile(asked, smoe::kPlaneTileSizes); }}
extern "C" int pair_tile(int asked) {{ return smoe::existing_tile(asked, smoe::kPairTileSizes); }}'''
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-shared", "-fPIC", "-x", "c++", "-", "-o", str(path)],
                   input=code, text=True, check=True)
    return ctypes.CDLL(str(path))


@pytest.mark.parametrize("asked,planes,pair", [(-2 ** 31, 0, 0), (-1, 0, 0), (0, 0, 0), (1, 16, 16), (8, 16, 16), (16, 16, 16), (17, 24, 32),
                                               (24, 24, 32), (25, 24, 32), (32, 24, 32), (33, 24, 64), (2 ** 31 - 1, 24, 64)])
def test_switch_selects_an_existing_size(lib, asked, planes, pair):
    assert lib.plane_tile(asked) == planes and lib.pair_tile(asked) == pair


def test_switches_are_read_through_it():
    text = open(os.path.join(CSRC, "api.cu")).read()
    for name, sizes in (("STRATA_MOE_PLANES_TILE", "kPlaneTileSizes"), ("STRATA_MOE_PAIR_NTILE", "kPairTileSizes")):
        assert f'existing_tile(num("{name}", 0), {sizes})' in text
