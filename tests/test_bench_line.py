"""The bench's result line stays short: an autotuner's candidates are counted in it, their times go to
stderr (a fake engine; no device needed)."""
import argparse
import json

import bench


class FakeEngine:
    def autotune(self, trials):
        return [{"pending_max": 8, "threads": 128, "us_per_trial": 0.5 * trials + k} for k in range(31)]


def test_autotune_times_go_to_stderr(capsys):
    assert bench.tune_engine(FakeEngine(), argparse.Namespace(tuning=None, quorum=None), 1000) == 31
    out, err = capsys.readouterr()
    assert out == ""
    assert len(json.loads(err.split("autotune: ", 1)[1])) == 31
