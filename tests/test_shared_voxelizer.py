"""voxelize_mesh_to_lattice from several threads: the calls share one engine, and each must
return its own grid.  The library is replaced by a fake that yields between its steps."""
import threading
import time

from aerosim_b200 import engine


def test_calls_of_several_threads_do_not_mix(monkeypatch):
    class Fake:
        made = 0

        def __init__(self, device):
            time.sleep(0.002)
            Fake.made += 1
            self.grid, self.inside = None, 0

    def voxelize_into(handle, geometry, world, tunnel, grid):
        handle.inside += 1
        assert handle.inside == 1, "two calls in the library at a time"
        handle.grid = grid["nx"]
        time.sleep(0.002)

    def read_voxel_grid(handle):
        time.sleep(0.001)
        handle.inside -= 1
        return handle.grid

    monkeypatch.setattr(engine, "_Handle", Fake)
    monkeypatch.setattr(engine, "_shared_voxelizer", None)
    monkeypatch.setattr(engine, "voxelize_into", voxelize_into)
    monkeypatch.setattr(engine, "read_voxel_grid", read_voxel_grid)
    got, errors = {}, []

    def work(k):
        try:
            for i in range(10):
                nx = 100 * k + i
                got[nx] = engine.voxelize_mesh_to_lattice(None, None, None, {"nx": nx, "ny": 1, "nz": 1})
        except BaseException as e:  # noqa: BLE001 - the test reports what a thread met
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and Fake.made == 1
    assert len(got) == 60 and all(k == v for k, v in got.items())
