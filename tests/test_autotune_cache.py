"""The autotuner's cache: an entry is taken for the library build that it was
measured with and for no other."""
import json
from types import SimpleNamespace

import pytest

from vk_gltf_viewer_gb300 import abi, autotune

SCENE = SimpleNamespace(host=SimpleNamespace(triangle_count=1000), draw_count=12)
VIEWS = [SimpleNamespace(width=640, height=360), SimpleNamespace(width=97, height=61)]


class Sweeper:
    device = 0

    def __init__(self):
        self.sweeps = 0

    def sweep(self, scene, views, flags, launches):
        self.sweeps += 1
        return [(8, 1, 2.0), (32, 4, 1.0)], (32, 4)


@pytest.fixture
def lib(tmp_path, monkeypatch):
    path = tmp_path / "lib.so"
    path.write_bytes(b"one build")
    monkeypatch.setattr(abi, "LIB_PATH", path)
    monkeypatch.setattr(autotune, "device_key", lambda device: "gpu")
    return path


def test_an_entry_holds_for_one_build(lib, tmp_path):
    r, path = Sweeper(), tmp_path / "tune.json"
    first = autotune.tune(r, SCENE, VIEWS, 3, path=path)
    assert not first["cached"] and r.sweeps == 1
    again = autotune.tune(r, SCENE, VIEWS, 3, path=path)
    assert again["cached"] and again["key"] == first["key"] and r.sweeps == 1
    lib.write_bytes(b"another build")
    other = autotune.tune(r, SCENE, VIEWS, 3, path=path)
    assert not other["cached"] and other["key"] != first["key"] and r.sweeps == 2
    assert set(json.loads(path.read_text())) == {first["key"], other["key"]}


def test_an_entry_without_a_build_is_swept_again(lib, tmp_path):
    r, path = Sweeper(), tmp_path / "tune.json"
    path.write_text(json.dumps({"gpu||" + autotune.workload_key(SCENE, VIEWS, 3):
                                {"bin_size": 8, "meshlets_per_cta": 1, "table": []}}))
    rec = autotune.tune(r, SCENE, VIEWS, 3, path=path)
    assert not rec["cached"] and (rec["bin_size"], rec["meshlets_per_cta"]) == (32, 4)
