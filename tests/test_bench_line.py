"""The line bench.py prints is read from the end of a log: with 64 realizations
and every leg it stays under 8 KB, and what the contract names is untouched."""
import json

import bench


def _full_line():
    text = "x" * 320
    err = {k: 1.2345678901234567e-5 for k in ("mean_disp_x_rel", "var_x_rel", "var_y_rel", "var_z_rel", "btc_l1_rel",
                                              "mc_var_rel_se")}
    err.update(btc_final=[434140, 434031], active=[744493, 744493])
    grad = {f"par{k}": {f"v{j}": 42473.971165541385 for j in range(5)} for k in range(10)}
    line = {k: 1.0283456789012345e9 for k in bench.CONTRACT}
    line.update(config={"workload": text, "flow_input": text}, roofline={"note": text, "achieved": 1234.5678901234567},
                e2e={"value": 1003914829.89327, "h2d_bytes_per_step": 64000000}, cpu_baseline={"sample": text})
    line.update(batched={"workload": text, "value": 9.876543210987654e9, "realizations": 64,
                         "error_vs_plain_fp64": {"worst_over_realizations": err, "per_realization": [err] * 64}},
                adjoint={"note": text * 3, "gradient_check": grad, "particle_steps": 1000000000},
                uniform_pulse={k: {"plume": [err] * 3} for k in ("fp64", "mixed")})
    return line


def test_line_is_short_and_keeps_the_contract():
    full = _full_line()
    line = bench.compact(full)
    text = json.dumps(line)
    assert len(json.dumps(full)) > 20000 and len(text) < 8000
    assert list(line) == list(full)
    for k in bench.CONTRACT:
        assert line[k] == full[k]
    b = json.loads(text)["batched"]
    assert b["realizations"] == 64 and b["value"] == 9.87654e9
    assert b["error_vs_plain_fp64"]["worst_over_realizations"]["active"] == [744493, 744493]
    assert "per_realization" not in b["error_vs_plain_fp64"]
