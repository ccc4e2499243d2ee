"""
What an SCF workspace holds: the digit planes only where they are used, one
fixed-point matrix without multipoles and ten with them.
"""

import ctypes as C

import pytest


@pytest.fixture(scope="module")
def L():
    from dxtb_gb300 import build

    lib = C.CDLL(str(build.build()))
    lib.dxtb_scf_workspace_mol.restype = lib.dxtb_scf_workspace_size.restype = C.c_int64
    lib.dxtb_scf_workspace_mol.argtypes = [C.c_int64] * 2
    lib.dxtb_scf_workspace_size.argtypes = [C.c_int64] * 2 + [C.c_int32] * 2
    return lib


@pytest.mark.parametrize("n,nat", [(1, 1), (12, 3), (13, 4), (16, 4), (17, 5), (354, 150), (5200, 2000)])
def test_workspace_sizes(L, n, nat):
    gfn1, gfn2 = (L.dxtb_scf_workspace_size(n, nat, mp, 1) for mp in (0, 1))
    bare = L.dxtb_scf_workspace_size(n, nat, 1, 0)
    assert L.dxtb_scf_workspace_mol(n, nat) == gfn2 and L.dxtb_scf_workspace_size(n, nat, 0, 0) == bare
    if n <= 12:
        assert gfn1 == gfn2 == bare
        return
    nb = (n + 15) // 16
    tiles = nb * (nb + 1) // 2
    assert gfn2 - gfn1 == tiles * (10 * 512 - 512)  # doubles: 10 matrices of pairs and mirrors, or S's pairs
    np2 = 256 * nb * nb
    assert gfn1 - bare >= 11 * np2 + 512 * tiles  # planes, vectors, S
    assert gfn1 - bare <= 11 * np2 + 512 * tiles + 200 * nb + 20 * n + 9 * nat + 256
