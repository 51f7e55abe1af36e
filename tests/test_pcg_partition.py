"""The PCG kernels' shared memory against their layouts, host only: for a mesh
split over the engine's grid, what the engine allocates covers what the kernel
addresses (restated here from the arrays that it keeps)."""
import ctypes

import numpy as np
import pytest


class Partition(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int) for n in ("ctas", "halo_max", "slot_max", "remote_max", "neighbour_max", "single_form",
                                             "global_parts")] + [
        (n, ctypes.c_longlong) for n in ("two_level_bytes", "single_bytes", "global_bytes")]


def partition(mesh, ctas=148, coord=True):
    from cbs3d import gpu
    L = gpu.lib()
    L.cbs3d_probe_pcg_partition.restype = ctypes.c_int
    P = ctypes.c_void_p
    xyz = np.ascontiguousarray(mesh.coord, dtype=np.float64)
    conn = np.ascontiguousarray(mesh.intma, dtype=np.int32)
    out = Partition()
    rc = L.cbs3d_probe_pcg_partition(conn.shape[0], xyz.shape[0], P(conn.ctypes.data), None,
                                     P(xyz.ctypes.data) if coord else None, ctas, ctypes.byref(out))
    assert rc == 0
    return out


# the sizes at which the tilings of four and eight rows per thread end, and
# grids of fewer CTAs, where the own rows are more of a halo
@pytest.mark.parametrize("shape,ctas", [((72, 72, 72), 148), ((74, 74, 74), 148), ((76, 76, 76), 148),
                                        ((61, 81, 83), 148), ((63, 63, 63), 128), ((48, 48, 48), 64), ((5, 5, 5), 148)])
def test_two_level_kernel_has_the_shared_memory_it_addresses(shape, ctas):
    from cbs3d import cases
    p = partition(cases.box_mesh(*shape), ctas)
    # z, inverse diagonal (8 bytes) and position (4) per halo entry; columns
    need = 20 * p.halo_max + 2 * p.slot_max
    need = (need + 15) // 16 * 16
    # the neighbours' rows of the coarse inverse, three coarse vectors, a correction per neighbour
    need += 8 * (p.neighbour_max * p.ctas + 3 * p.ctas + p.neighbour_max)
    need += p.halo_max   # every entry's owner
    assert p.two_level_bytes >= need


# thin meshes and orders without coordinates, whose halos are mostly remote
@pytest.mark.parametrize("shape,coord", [((900, 16, 16), True), ((64, 64, 64), False), ((66, 66, 66), False),
                                         ((64, 64, 64), True)])
def test_single_reduction_kernel_has_a_form_that_fits(shape, coord):
    from cbs3d import cases
    p = partition(cases.box_mesh(*shape), 148, coord)
    assert p.single_form == (0 if coord and shape[0] == 64 else 1)
    # z per halo entry; per remote entry r, s and, in the first form, inverse
    # diagonal, position (4) and place (2); columns
    need = 8 * p.halo_max + (30 if p.single_form == 0 else 16) * p.remote_max + 2 * p.slot_max
    assert need <= p.single_bytes <= 220 * 1024


# two CTAs (or three): many slices each, and halos of one part fewer that fit
# without the slice table (216,352 bytes and a table of 15,632 at 49^3)
@pytest.mark.parametrize("n,ctas,parts", [(49, 2, 7), (51, 2, 8), (53, 3, 6), (48, 2, 6)])
def test_global_vector_kernel_counts_its_slice_table(n, ctas, parts):
    from cbs3d import cases
    p = partition(cases.box_mesh(n, n, n), ctas)
    assert p.global_parts == parts
    assert p.global_bytes <= 227 * 1024 - 2064   # the SM's limit less the kernel's static shared memory
