"""Slab inputs with relaxation values: uniform ones pass through, voxel maps are cut to the slab."""
import numpy as np

from mrsim_acq_b200 import shard
from mrsim_acq_b200.api import T2


def test_slab_inputs_cut_the_maps():
    nz, plane, nv = 4, 6, 2
    vox = np.arange(nz * plane, dtype=np.float32)
    t2 = [T2.uniform(80.0), T2.of_map(vox)]
    d = shard.slab_inputs((3, 2, nz), (3, 2, nz), nv, [np.zeros(nz * plane * nv, np.float32)], vox, 1, 3, t2, [T2.of_map(2 * vox)])
    assert d["t2"][0].value == 80.0 and d["t2"][0].map is None
    assert np.array_equal(d["t2"][1].map, vox[plane:3 * plane])
    assert np.array_equal(d["t_inhom"][0].map, 2 * vox[plane:3 * plane])
    assert np.array_equal(d["fmap"], vox[plane:3 * plane]) and d["slice_z"] == [1, 2]
