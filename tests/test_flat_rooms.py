"""The estimate pass's form of rooms (CPU: flat_scene, and the device functions
compiled as host code).  A room whose six walls bound a box exactly is no box
to trace from outside: every ray would start in it and be left to the exact
tests."""
import device_source


def test_rooms_are_not_boxes(tmp_path):
    rows = {}
    for line in device_source.run(tmp_path, "flat_rooms.cpp").splitlines():
        name, *v = line.split()
        rows[name] = dict(zip(("ok", "rects", "boxes", "rays", "doubt", "wrong", "s_doubt", "s_wrong"), map(int, v)))
    for name, r in rows.items():
        assert r["wrong"] == 0 and r["s_wrong"] == 0, name
    form = {name: (r["ok"], r["rects"], r["boxes"]) for name, r in rows.items()}
    assert form == {"closed": (1, 7, 0), "closed-furnished": (1, 7, 1), "closed-seen-from-outside": (1, 7, 0),
                    "box": (1, 1, 1), "lit-box": (1, 1, 1), "closed-turned": (0, 0, 0)}
    for name in ("closed", "closed-furnished", "closed-seen-from-outside"):
        r = rows[name]
        # the furnished room's box holds 1.5 of its 96 units of volume
        assert r["doubt"] < 0.03 * r["rays"] and r["s_doubt"] < 0.03 * r["rays"], (name, r)
