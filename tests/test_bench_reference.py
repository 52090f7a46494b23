"""The benchmark's host baseline where no build of the reference is present."""
import json
from types import SimpleNamespace

import bench
from oracle import pyoracle as po, ref_gpu


def test_reference_arm_without_the_reference_build(monkeypatch, capsys):
    """The oracle's restatement stands in for it and every step deposits."""
    monkeypatch.setattr(po, "ref_available", lambda *a: False)
    monkeypatch.setattr(ref_gpu, "available", lambda *a: False)
    monkeypatch.setattr(bench, "WORKLOAD", dict(bench.WORKLOAD, half_length_y1=10.0, half_length_y2=10.0,
                                                num_pixels_y1=10, num_pixels_y2=10, expansion_order=6))
    deposited = []
    deposit = po.ipm_deposit_ref
    monkeypatch.setattr(po, "ipm_deposit_ref", lambda *a: deposited.append(deposit(*a).sum()))
    bench.reference_arm(SimpleNamespace(steps=2, warmup=1, gpus=1))
    line = json.loads(capsys.readouterr().out)
    assert line["cpu_baseline"]["kind"] == "port" and line["steps"] == 2 and line["value"] > 0
    # the last call is the whole lattice: the mean magnification is that of the lens, to the field's scatter
    assert 3 < deposited[-1] / 10 ** 2 < 15
