"""CPU model of k_matvec_h8m's 32-bit byte offsets: a CTA counts them from its z
chunk's first plane, and the chunks are cut so that every plane it reads lies within
2^32 bytes of it, on grids whose vectors are larger than that."""
import pytest


def most_planes(sx, sy, size):
    return min((1 << 32) // (sx * sy * size), 1 << 30) - 3


def zchunk(sz, tiles, resident, most):
    best, cost, bz, zc = sz, None, 1, 0
    while zc != 1:
        zc = -(-sz // bz)
        if zc <= most:
            n = tiles * -(-sz // zc)
            c = -(-n // resident) * (zc + 1)
            if cost is None or c < cost:
                best, cost = zc, c
        bz = -(-sz // max(zc - 1, 1))
    return best


@pytest.mark.parametrize("size", [4, 8])
@pytest.mark.parametrize("nodes", [(2, 2, 2), (385, 129, 129), (821, 821, 811), (1025, 1025, 1025),
                                   (66000, 65, 65), (65, 65535, 200), (3, 3, 65535),
                                   (10001, 10001, 9), (11500, 11500, 5)])
def test_every_offset_fits_32_bits(nodes, size):
    sx, sy, sz = nodes
    most = most_planes(sx, sy, size)
    if most < 1:  # the dense kernel's: planes of more than 2^30 bytes
        assert sx * sy * size > 1 << 30
        return
    for rows in (8, 12):
        for resident in (148, 296, 444):
            zc = zchunk(sz, -(-sx // 31) * -(-sy // (rows - 1)), resident, most)
            seen = 0
            for z0 in range(0, sz, zc):
                z1 = min(z0 + zc, sz) - 1
                base = max(z0 - 1, 0)
                top = min(z1 + 1, sz - 1)  # planes base .. top are read, z0 .. z1 written
                assert base <= z0 and ((top - base + 1) * sx * sy) * size <= 1 << 32
                seen += z1 - z0 + 1
            assert seen == sz
