"""bench.py --impl reference: figures of anything but the reference's own core are
marked as such."""

import argparse


def test_without_the_reference_the_arm_says_so(monkeypatch):
    import bench
    from oracle import binding as O

    monkeypatch.setattr(O, "ref_available", lambda: False)
    res = bench.run_reference(argparse.Namespace(warmup=0, steps=1), 0, 1)
    assert res["impl"] == "reference" and "\n" not in res["unavailable"] and res["unavailable"]
    assert res["cpu_baseline"]["kind"] == "port"
