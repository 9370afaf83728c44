"""Host-only: what a Voronoi system needs per cell. 16-slot rows and their staging 136 bytes, queues and
claims 52, positions, preferences, motility, directors, forces, areas and perimeters 88, cell list 28 and
1 / 0.64 bins of 8, noise and the staged integration 16, indices and flags 12: 332 + 12.5 (the kept old
rows are bounded and add nothing here)."""


def test_bytes_per_cell(cglib):
    import ctypes as C

    size = lambda n: cglib.cg_voronoi_footprint(1, C.byref(C.c_int(n)), 16)
    per_cell = (size(4000000) - size(2000000)) / 2000000
    assert abs(per_cell - (332 + 8 / 0.64)) < 1.0
