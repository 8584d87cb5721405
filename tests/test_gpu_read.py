"""Reads into page-locked memory (k_gather_xyz writes there itself, whole quads of
words where the array is aligned for them): the same values as reads into ordinary
memory, at every alignment of the array and length of the last block, and no word
beyond it."""
import ctypes as C

import numpy as np
import pytest

import xfem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (7, 3, 7), (16, 14, 1), (5, 6, 6), (21, 9, 13)])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_page_locked_reads(dims, offset):
    meshes = [xfem.generate_tet_block(*d, (0.1, 0.1, 0.1), 0, 0.2) + (1000.0,) for d in (dims, (2, 2, 2))]
    b = xfem.Body(meshes=meshes, settings=[xfem.default_settings()] * 2)
    b.step_frames(1, 3, 1.0 / 1200.0)
    for k in range(2):
        n = 3 * b.counts[k][0]
        p = xfem.lib().xfem_alloc_host((n + 8) * 4)
        try:
            a = np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), (n + 8,))
            for read in (b.positions, b.velocities):
                a[:] = -7.0
                read(k, out=a[offset:offset + n])
                assert np.array_equal(a[offset:offset + n].reshape(-1, 3), read(k))
                assert np.all(a[:offset] == -7.0) and np.all(a[offset + n:] == -7.0)
        finally:
            xfem.lib().xfem_free_host(p)
