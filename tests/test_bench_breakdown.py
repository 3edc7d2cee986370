"""bench.py's kernel breakdown times what the timed step runs."""
import bench


class _Event:
    def __init__(self, enable_timing=False):
        pass

    def record(self, stream):
        pass

    def synchronize(self):
        pass

    def elapsed_time(self, other):
        return 12.0


class _Sim:
    def __init__(self):
        self.calls = set()

    def __getattr__(self, name):
        return lambda *a: self.calls.add(name)


def test_breakdown_of_the_shared_memory_free_step(monkeypatch):
    import torch
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    own = dict(kernels=3, tile_x=30, tile_y=10, zchunk=64, threads=0)
    V = 512 ** 3
    assert bench.steps_without_shared_memory(own, own, True, V)
    assert not bench.steps_without_shared_memory(dict(own, zchunk=32), own, True, V)
    assert not bench.steps_without_shared_memory(own, own, False, V)
    assert not bench.steps_without_shared_memory(own, own, True, 1024 ** 3)
    sim = _Sim()
    k = bench.kernel_breakdown(sim, "point", "fp32", V, None, 4, 512 * 512, True)
    assert sim.calls == {"step"}  # not the two stages apart, which other kernels run
    # update: 8 words in, 14 out; LBM: 15 populations in and out, 9 words in, 3 out
    assert k == {"point_step": {"ms": 3.0, "bytes_per_cell": 4 * (8 + 14 + 30 + 9 + 3)}}
    for kernels in ("split", "split_pair"):
        sim = _Sim()
        assert set(bench.kernel_breakdown(sim, kernels, "fp32", V, None, 4)) == {"qforce", "lbm"}
        assert sim.calls == {"step", "qtensor_step", "lbm_step"}
