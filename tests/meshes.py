"""Tetrahedral boxes whose rows are wider than the Kuhn mesh's fourteen
neighbours: the five-tetrahedra split (rows of 6 and 18) and the
24-tetrahedra split with face and cube centres (rows of 6, 14 and 26)."""
import numpy as np

from cbs3d import cases


def _mesh(coord, intma, shape):
    """The cases' Mesh of a unit box from its nodes and tetrahedra (0-based)."""
    x = coord[intma]
    vol6 = np.einsum("ij,ij->i", x[:, 1] - x[:, 0], np.cross(x[:, 2] - x[:, 0], x[:, 3] - x[:, 0]))
    intma = np.where((vol6 < 0)[:, None], intma[:, [0, 2, 1, 3]], intma)
    faces = []
    for fn in cases._FACE_NODES:
        tri = intma[:, list(fn)]
        for plane in range(6):
            on = np.all(coord[tri][:, :, plane // 2] == plane % 2, axis=1)
            e = np.nonzero(on)[0]
            faces.append(np.column_stack([tri[e] + 1, e + 1, np.full(e.size, plane + 1)]))
    bf = np.concatenate(faces)
    bf = bf[np.argsort(bf[:, 3], kind="stable")].astype(np.int32)
    return cases.Mesh(coord=coord, intma=(intma + 1).astype(np.int32), bfaces=bf, lattice=None, shape=shape,
                      mat_elem=np.zeros(intma.shape[0], dtype=np.int32))


def _lattice(nx, ny, nz):
    k, j, i = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
    lat = np.stack([i.ravel(), j.ravel(), k.ravel()], axis=1)
    cube = lat[(lat[:, 0] < nx) & (lat[:, 1] < ny) & (lat[:, 2] < nz)]
    return lat, cube, lambda p: p[..., 0] + (nx + 1) * (p[..., 1] + (ny + 1) * p[..., 2])


def five_tet_box(nx, ny, nz):
    lat, cube, nid = _lattice(nx, ny, nz)
    corners = np.array([(a, b, c) for c in (0, 1) for b in (0, 1) for a in (0, 1)])
    tets = []
    for parity in (0, 1):
        c = cube[cube.sum(axis=1) % 2 == parity]
        inner = [v for v in corners if v.sum() % 2 == parity]
        split = [inner] + [[v] + [np.where(np.arange(3) == d, 1 - v, v) for d in range(3)]
                           for v in corners if v.sum() % 2 != parity]
        for t in split:
            tets.append(np.stack([nid(c + v) for v in t], axis=1))
    return _mesh(lat / np.array([nx, ny, nz], dtype=float), np.concatenate(tets), (nx, ny, nz))


def centred_box(nx, ny, nz):
    lat, cube, nid = _lattice(nx, ny, nz)
    coords, first, ids = [2 * lat], lat.shape[0], {}
    tets = []
    centre = first + np.arange(cube.shape[0])
    coords.append(2 * cube + 1)
    first += cube.shape[0]
    for d in range(3):
        lo = lat[np.all((lat < np.array([nx, ny, nz])) | (np.arange(3) == d), axis=1)]
        num = np.full(lat.shape[0], -1)
        num[nid(lo)] = first + np.arange(lo.shape[0])
        first += lo.shape[0]
        coords.append(2 * lo + (np.arange(3) != d))
        ids[d] = num
    for d in range(3):
        ring = np.zeros((4, 3), dtype=int)
        ring[:, [a for a in range(3) if a != d]] = ((0, 0), (1, 0), (1, 1), (0, 1))
        for side in (0, 1):
            base = cube + side * (np.arange(3) == d)
            for q in range(4):
                tets.append(np.stack([centre, ids[d][nid(base)], nid(base + ring[q]), nid(base + ring[(q + 1) % 4])], axis=1))
    coord = np.concatenate(coords) / (2.0 * np.array([nx, ny, nz]))
    return _mesh(coord, np.concatenate(tets), (nx, ny, nz))


def cavity(mesh, re=400.0, **over):
    """The lid-driven cavity on one of these boxes."""
    p = cases.default_params(re=re, ntime=10 ** 6, pnode=1, inlet_u=1.0, inlet_v=0.0, inlet_w=0.0, **over)
    return cases.Case(mesh=mesh, bc_map=dict(cases.CAVITY_BC), params=p)
