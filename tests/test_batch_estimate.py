"""The device bytes that the batch engine reserves for a solve's XC buffers cover
what a group of chunks holds: AO values, gradients and weighted AOs (40 bytes a
function and point, 256 MB a group), the P block and the slices of V of every
chunk in it, and the V accumulators, on each XC stream."""

from ctypes import byref, c_int64

import numpy as np
import pytest


def _estimate(mol, streams, chunk, npoint):
    from dftax_b200 import _lib
    from dftax_b200.batch import make_request

    sym, xyz, orb, aux, _ = mol
    r, keep, _ = make_request(sym, xyz, orb, aux, grid=(np.zeros((npoint, 3)), np.zeros(npoint)),
                              scf_opts={"xc_streams": streams, "grid_chunk": chunk})
    b = c_int64()
    _lib.check(_lib.load().dfbatch_estimate(byref(r), byref(b)))
    return b.value


@pytest.mark.parametrize("name", ["water", "water5", "alkane10"])
@pytest.mark.parametrize("chunk", [0, 256, 512, 8192])
def test_a_stream_covers_its_group(name, chunk):
    from dftax_b200 import systems

    mol = systems.workload(name, seed=0)
    nao, npoint = mol[2].nao, 200000
    per_stream = (_estimate(mol, 8, chunk, npoint) - _estimate(mol, 1, chunk, npoint)) / 7
    for G in [chunk] if chunk else [512, 1024, 2048, 4096, 8192, 16384]:
        chunks = -(-npoint // G)
        for nsig in (1, nao // 4, nao // 2, nao):   # functions of every chunk
            count = min(chunks, max(1, (256 << 20) // (40 * nsig * G)))
            blocks = 8 * count * (nsig * (nsig + 1) + -(-G // 512) * nsig * nsig)
            need = count * (40 * nsig + 32) * G + blocks + 8 * nao * nao
            assert per_stream >= need, (G, nsig)


def test_a_small_grid_fills_no_group():
    """One water with 28000 points holds 34 MB of AO planes: its request fits a budget
    of 400 MB, 256 of which the estimate always keeps."""
    from dftax_b200 import systems

    assert _estimate(systems.workload("water", seed=0), 1, 0, 28000) < 400 << 20
