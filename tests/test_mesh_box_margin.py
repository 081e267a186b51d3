"""The mesh's box test before a BVH walk, from any distance (CPU: the device
functions compiled as host code)."""
import device_source


def test_no_ray_of_the_walk_is_turned_away(tmp_path):
    rows = [line.split() for line in device_source.run(tmp_path, "mesh_box.cpp").splitlines()]
    assert len(rows) == 5
    for dist, met, lost in rows:
        assert int(met) > 50_000, dist
        assert int(lost) == 0, f"{lost} of {met} rays lost at distance {dist}"
