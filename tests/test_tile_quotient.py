"""The integer quotient of the tile kernels (seis_b200/csrc/fd_tile.cuh, quot):
(i + 0.5) r rounded down is i / len for every i below 2^13 and every column
length up to a tile's 128 rows and its halo's two, with r = 1 / len rounded to
nearest and two units in the last place off either way (the contracted build's
division)."""
import numpy as np


def test_quotient_of_every_index_and_length():
    i = np.arange(1 << 13)
    x = i.astype(np.float32) + np.float32(0.5)
    for n in range(1, 131):
        r = np.float32(1.0) / np.float32(n)
        ulp = np.spacing(r)
        for k in (-2, -1, 0, 1, 2):
            q = (x * np.float32(r + k * ulp)).astype(np.int32)
            assert np.array_equal(q, i // n), (n, k)
