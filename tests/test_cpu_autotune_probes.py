"""The batched-launch autotuner tries only knobs that its probes depend on, and its table names the probes."""
import json
import os

from krans_b200 import autotune as T


def test_lanes_are_not_tried_on_operands_that_do_not_use_them():
    tried = [name for name, _ in T.PROBED]
    assert tried == ["cluster_size", "cluster_min", "pair_max"]
    _, _, trials = T.search(lambda k: 100.0, T.DEFAULTS, T.PROBED)
    assert all(t["knobs"]["lanes"] == T.DEFAULTS["lanes"] for t in trials)


def test_stored_tables_name_their_probe_batches():
    for f in os.listdir(T.TABLE_DIR):
        with open(os.path.join(T.TABLE_DIR, f)) as fh:
            batches = json.load(fh)["probe"]["batches"]
        assert batches and all({"count", "seed", "n_hi"} <= set(b) for b in batches)
