"""One HeldSuarezPhysics over several grids: each gets the table of its own latitudes, also where a
grid is gone before the next is made (whose object may then have the old one's address), and where
a grid's latitudes are replaced in place."""
import importlib

import numpy as np

pkg = importlib.import_module("jax-gcm_b200")
H = importlib.import_module("jax-gcm_b200.held_suarez")


def want(lat):
    la = np.asarray(lat, np.float64).astype(np.float32)
    return np.stack([np.sin(la) ** 2, np.cos(la) ** 2, np.cos(la) ** 4]).astype(np.float32)


def test_tables_follow_the_latitudes():
    phys = pkg.HeldSuarezPhysics()
    for _ in range(3):
        for ix, il in ((128, 64), (95, 47), (256, 128), (12, 64)):
            lat = np.linspace(-1.4, 1.4, il) + 0.001 * ix
            geom = pkg.Geometry.from_grid_shape((ix, il), 8, latitudes=lat, device="cpu")
            tab = phys._lat_table(geom, "cpu")
            assert np.array_equal(tab.numpy(), want(lat)), (ix, il)
            assert phys._lat_table(geom, "cpu") is tab
            del geom


def test_replaced_latitudes():
    phys = pkg.HeldSuarezPhysics()
    geom = pkg.Geometry.from_grid_shape((8, 16), 8, device="cpu")
    phys._lat_table(geom, "cpu")
    geom.radang = np.linspace(-1.0, 1.0, 16)
    assert np.array_equal(phys._lat_table(geom, "cpu").numpy(), want(geom.radang))
