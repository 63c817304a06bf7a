"""bench.py's transport line names a kernel only with a time that is its own: the
reconstruction kind holds two kernels (18 launches of the partial cells' fluxes
and 6 of the normals), whose times are summed."""
import json
import sys
import types

from test_transport_host import ROOT, _BenchHostLib, host_lib  # noqa: F401


class _SlowReconstruction(_BenchHostLib):
    def scf_clsvof_run(self, ctx, steps, pstats):
        super().scf_clsvof_run(ctx, steps, pstats)
        if self.timing:
            pstats._obj.ms_kernels[:] = [2.4 * steps, 0.9 * steps, 0.01 * steps, 0.2 * steps]
        return 0


def test_roofline_is_that_of_one_kernel(host_lib, monkeypatch, capsys):  # noqa: F811
    sys.path.insert(0, ROOT)
    import bench
    from simcoflow3d_gb300 import projection
    monkeypatch.setattr(projection, "load_library", lambda: _SlowReconstruction(host_lib))
    assert bench.run_clsvof(types.SimpleNamespace(n=16, warmup=3, steps=2, no_cpu=True, seed=1)) == 0
    rf = json.loads(capsys.readouterr().out.strip().splitlines()[-1])["roofline"]
    assert rf["kernel"] == "k_sweep" and rf["ms_per_launch"] == 0.9 / 18
    assert rf["bytes_per_launch"] == 16 ** 3 * (40 + 2 * 56) // 3
    assert abs(rf["achieved"] - 6 * 16 ** 3 * (40 + 2 * 56) / 0.9e-3 / 1e9) <= 0.051   # printed to 0.1
    assert rf["kinds_ms_per_step"]["reconstruct"] == 2.4
    assert rf["kinds_launches"] == {"reconstruct": "18 k_partial_fluxes, 6 k_normals", "sweep": "18 k_sweep",
                                    "walls": "6 k_walls", "redistance": "6 each of k_band_bound, k_band_pairs, k_band_value"}
