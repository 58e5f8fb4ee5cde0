"""The benchmark's printed line."""
import json

import bench


def test_default_line_stays_short():
    """The other configurations, lists over 64 instances and all, leave a line
    that fits the last 3,000 characters of the output; the headline's own keys
    are untouched, and nothing is lost."""
    head = {"metric": "Gibbs tokens/sec (LDA)", "value": 5232785291.391, "config": {"workload": "w" * 250}, "roofline": {"note": "n" * 580},
            "e2e": {"note": "e" * 290}, "rest": "r" * 600}
    inst = {"N": 81448, "D": 256, "rounds": 340, "min_ess": 1463.0833157454445, "min_ess_per_s": 466.8766343822553}
    other = {"hlr_nuts": {"value": 104.8989310462663, "unit": "min-ESS/s", "seconds": 3.1337685546875, "gain_vs_cpu_core": 26925.812895700026,
                          "instances": [inst] * 64},
             "gmm": {"value": 444513988.1898497, "unit": "points/s", "ms_per_sweep": 0.44992959797382354, "config": {"N": 200000}},
             "hlr_small": {"value": 24192.76, "unit": "min-ESS/s", "chains": 256, "gain_single_chain_vs_cpu": 8.7, "batched": {"ms": 66.4}},
             "hlr_surrogate": {"value": 1106.9, "unit": "min-ESS/s", "gain_vs_plain": 17.8, "ms_per_iteration": {"plain": 29.55888671875},
                               "posterior_mean_diff_in_sd": 0.0139, "fallback": False, "exactness": {"iterations": {"plain": 1000}}}}
    line, full = bench.brief(dict(head, **other))
    assert len(json.dumps(line)) < 2900
    assert all(line[k] == v for k, v in head.items())
    assert full == other
    assert line["gmm"] == {"value": 444514000.0, "unit": "points/s", "ms_per_sweep": 0.44993}
    assert line["hlr_surrogate"]["ms_per_iteration"] == {"plain": 29.5589}
    assert bench.brief(head) == (head, {})
    assert bench.brief({"gmm": {"error": "x"}})[0] == {"gmm": {"error": "x"}}
