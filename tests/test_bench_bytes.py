"""The bytes that bench.py counts for the distance transform, on masks whose
planes with sources and columns with targets can be counted by hand."""
import numpy as np
import torch

import bench


def masks(*voxels, shape=(40, 50, 100)):
    out = []
    for vs in voxels:
        m = np.zeros(shape, np.uint8)
        for v in vs:
            m[v] = 1
        out.append(torch.from_numpy(m))
    return out


def test_two_far_voxels():
    # domain: planes 2..37 (36), rows 3..44 (42), words 0..2; one plane with a source and one column each way
    a, b = masks([(2, 3, 4)], [(37, 44, 90)])
    assert bench._transform_bytes(a, b) == 2 * (42 * 96 + 4 * 32)


def test_planes_and_columns():
    # domain: rows 10..17, words 1..2.  A has planes 1, 2 and 5, B plane 5 only; B's voxels outside A lie in the columns
    # (rows 10 - 13, word 2) and (rows 14 - 17, word 1), A's outside B in (rows 10 - 13, word 1)
    a, b = masks([(1, 10, 40), (2, 11, 41), (5, 12, 63)], [(5, 10, 64), (5, 14, 33), (5, 17, 33), (5, 12, 63)])
    assert bench._transform_bytes(a, b) == 3 * (8 * 64 + 2 * 4 * 32) + 1 * (8 * 64 + 1 * 4 * 32)


def test_nothing_to_measure():
    a, b = masks([(1, 10, 40)], [])
    assert bench._transform_bytes(a, b) == bench._transform_bytes(b, b) == bench._transform_bytes(a, a) == 0
