"""The room for a reduction's partial sums (nereus_b200_sum_blocks, host only) against the launch grids of the kernels
that end in a grid-wide sum, restated here, over grids up to the 2^31 cells a layout may have."""
import random

import pytest

from nereus_cfd_b200 import capi

SLOTS = (148, 148 * 8)  # resident blocks of a launch: one to eight a multiprocessor


def up(a, b):
    return -(-a // b)


def quad_blocks(Nx, Ny, Nz, n, slots):
    """A quad kernel of n elements a thread: the longest march of at most 16 planes that fills its last wave to 90%,
    else the one that fills it best."""
    per = up(Nx * (up((Nz + 1) // 2, 4) * 4 // n), 256)
    best = None
    for S in range(16, 0, -1):
        blocks = per * up(Ny - 2, S)
        fill = blocks / (up(blocks, slots) * slots)
        if fill >= 0.9:
            return blocks
        if best is None or fill > best[0]:
            best = (fill, blocks)
    return best[1]


def grids(dim, Nx, Ny, Nz):
    """Blocks of every such launch on level 0."""
    if dim == 2:
        # a thread per cell in tiles of 32 x 8, and the fused ascent's blocks of 32 x 16
        yield up(Nx - 2, 32) * up(Ny - 2, 8)
        yield up(Nx - 2, 32) * up(Ny - 2, 16)
        return
    per = up(Nz - 2, 32) * up(Nx - 2, 8)
    yield per * up(Ny - 2, max(1, min(up((Ny - 2) * per, 148 * 16), Ny - 2)))
    pairs = up(Nx * ((Nz + 1) // 2), 256)
    march = max(min(16, Ny - 2), min(8, max(1, up((Ny - 2) * pairs, 148 * 8))))
    yield pairs * up(Ny - 2, march)
    for n in (2, 4):
        for slots in SLOTS:
            yield quad_blocks(Nx, Ny, Nz, n, slots)
    if Nx * Ny * Nz <= 300000:  # the legs of small levels: a block for 4 x 4 x 8 coarse cells
        yield up(up(Nz - 2, 2), 8) * up(up(Nx - 2, 2), 4) * up(up(Ny - 2, 2), 4)


def check(dim, Nx, Ny, Nz):
    room = capi.load().nereus_b200_sum_blocks(dim, Nx, Ny, Nz)
    need = max(grids(dim, Nx, Ny, Nz))
    assert room >= max(need, 65536), (dim, Nx, Ny, Nz, room, need)
    return need


# 810^3 and 1024^3 interior cells: more than 65536 blocks in the refinement step's two sums and the half-sweep's three;
# a slab; 4100^2 and 46000^2 in two dimensions
@pytest.mark.parametrize("size", [(3, 812, 812, 812), (3, 1026, 1026, 1026), (3, 1023, 1291, 1024), (3, 4200, 10, 4200),
                                  (2, 4102, 4102, 1), (2, 46000, 46000, 1)])
def test_large_grids_have_room(size):
    assert check(*size) > 65536


def test_random_sizes_have_room():
    rng = random.Random(5)
    for _ in range(3000):
        dim = rng.choice((2, 3))
        while True:
            n = [int(3 * 2 ** rng.uniform(0, 17)) for _ in range(dim)] + [1] * (3 - dim)
            if n[0] * n[1] * n[2] < 2 ** 31:
                break
        check(dim, *n)


def test_bad_sizes_are_refused():
    lib = capi.load()
    for size in ((1, 8, 8, 8), (3, 1, 8, 8), (3, 8, 8, 1), (2, 8, 1, 1)):
        assert lib.nereus_b200_sum_blocks(*size) == capi.NB_BAD_INPUT
