"""The benchmark's printed line: every key of the contract as recorded, without the sweeps that make the record long."""
import json


def test_printed_line_is_short_and_keeps_the_contract():
    import bench

    contract = dict(metric=bench.METRIC, value=1.0, unit="queries/s", n_gpus=1, steps=3, warmup=3, ms_per_step=1.0,
                    higher_is_better=True, scaling="weak", vs_baseline=None, dtype="f32", data="synthetic",
                    config=bench.CONFIG, e2e=dict(value=1.0, unit="queries/s", h2d_bytes_per_step=1, d2h_bytes_per_step=2),
                    gpu_launches=4, clocks=dict(sm_mhz=1965.0, sm_max_mhz=1965.0, reasons=[]))
    form = dict(beam=45, recall_at_10=0.95, qps_batched_graph=1.0, speedup_vs_plain=1.1,
                scoring_error_vs_fp64=dict(pairs=40000, abs_max=0.1))
    sweep = [dict(k=10, beam=b, recall=0.9, qps=1.0) for b in range(120)]
    line = dict(contract, details=dict(beam=45, recall_sweep=[[b, 0.9] for b in range(40)]),
                forms=dict(precision_batched={f"bf16_{i}": dict(form, qps_batched_graph=i) for i in range(8)},
                           range=dict(qps_e2e=10.4), search_and_parse=dict(runs=sweep)))
    out = bench.printed(line)
    assert {k: out[k] for k in contract} == contract
    assert out["details"] == dict(beam=45)
    assert out["forms_qps"] == {"precision_batched": 7, "range": 10}
    assert len(json.dumps(out)) < 2600 < len(json.dumps(line))
    assert line["details"]["recall_sweep"], "the record itself stays whole"
