"""The bench's printed line: every figure of the result, none of the tables,
and short enough to be kept whole by a reader of the run's last output."""
import json
import types

import bench


def _result():
    third = 1.0 / 3.0
    table = {str(th): {"rms_err": 0.0028886512345678, "rms_rel_err_per_vertex": third,
                       "max_err_over_rms_force": third} for th in bench.LEARNED_THETAS}
    learned = {"train_s": 47.038312345678, "train_pairs": 12585989,
               "train_loss_first_last": [third, third], "judge_vertices": 1048576,
               "plain_rms_err": third, "plain_rms_rel_err_per_vertex": third,
               "plain_max_err_over_rms_force": third, "learned_theta": 1.225,
               "hub_targets": 1024, "hub_theta": 0.35, "learned_errors": table,
               "plain_errors": table, "hub_choice": "auto",
               "candidates": [{"hub_targets": k, "theta": 1.225, "ms_per_step": 1 + third,
                               "rms_err": third} for k in (0, 1024, 4096)],
               "learned_errors_by_hub_targets": {k: table for k in ("0", "1024", "4096")},
               "group_spread": 1.0, "walk": "cell groups", "value": 752 + third,
               "theta": 1.225, "rms_err": third}
    kernels = {k: 0.1234 for k in ("tree_keys", "radix_sort", "tree_buckets", "tree_nodes",
                                   "attraction_f32", "bh_walk_f32_learned", "bh_walk_hubs",
                                   "fa2_update")}
    w = bench.Workload.__new__(bench.Workload)
    w.name = "ba1m_learned"
    return {"metric": w.metric(), "value": 752 + third, "unit": "iters/s", "n_gpus": 1,
            "steps": 20, "warmup": 5, "ms_per_step": 1 + third, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": "ba1m_learned: barabasi_albert n=1048576 m=4 edges=4194294",
                       "model": "linlog", "theta": {"plain": 0.5, "learned": 1.225},
                       "barnes_hut": True, "gravity": 1.0, "overlap_radius": None, "graphs": 1,
                       "vertices": 1048576, "seed": 7, "precision": "fp32-walk",
                       "parallelism": "replicas1", "hub_targets": 1024,
                       "l2": "per-step working set > L2 (tree rebuilt every step)"},
            "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"],
                       "samples": 500},
            "e2e": {"value": 542 + third, "unit": "iters/s", "h2d_bytes_per_step": 16777216,
                    "d2h_bytes_per_step": 16777216, "steps": 20, "timer": "t" * 240},
            "gpu_launches": 480, "kernels_per_step": 24, "vertex_updates_per_s": 1e9 * third,
            "roofline": {"kernel": "bh_walk_f32_learned", "bound": "tensor", "achieved": third,
                         "peak": 1661.8, "unit": "TFLOP/s", "frac": third, "traffic": 873e6,
                         "traffic_source": "s" * 70, "peak_source": "s" * 90,
                         "algorithmic": "a" * 120, "share_of_step": third,
                         "warp_node_visits": 9051228,
                         "fp32_view": {"achieved": third, "peak": third, "frac": third,
                                       "algorithmic": "a" * 90}},
            "kernel_ms": kernels, "peaks": "measured", "walk_shape": {"threads": 64},
            "learned": learned,
            "plain": {"theta": 0.5, "value": third, "ms_per_step": third, "rms_err": third,
                      "kernel_ms": kernels, "interactions": 333189242,
                      "warp_node_visits": 22401905, "walk_fp32_frac": third,
                      "walk_traffic": 783.2e6},
            "cpu_baseline": {"value": third, "unit": "iters/s", "cores": 16, "kind": "port",
                             "cpu_model": "c" * 60, "sample": "s" * 110}}


def test_line_is_short_and_keeps_every_figure():
    full = _result()
    got = bench.brief(full)
    text = json.dumps(got)
    assert len(json.dumps(full)) > 10000 and len(text) < 3000
    for k, v in full.items():
        if not isinstance(v, dict):
            assert got[k] == v  # the contract's figures, unrounded
    assert set(full) - set(got) == {"walk_shape"}
    for part in ("config", "clocks", "e2e", "kernel_ms", "cpu_baseline", "plain", "roofline"):
        for k, v in full[part].items():
            if k in bench.LONG_KEYS or isinstance(v, dict):
                continue
            same = got[part][k] == v
            assert same or abs(got[part][k] - v) <= 1e-5 * abs(v)
    assert got["learned"]["candidates"][1]["hub_targets"] == 1024


def test_details_file_has_everything(tmp_path, capsys):
    full = _result()
    bench.print_line(full, types.SimpleNamespace(details=str(tmp_path / "d.json")))
    out = capsys.readouterr().out
    assert out.count("\n") == 1 and json.loads(out)["metric"] == full["metric"]
    assert json.load(open(tmp_path / "d.json")) == json.loads(json.dumps(full))
    bench.print_line(full, types.SimpleNamespace(details=None))
    assert len(capsys.readouterr().out) < 3000
