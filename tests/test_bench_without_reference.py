"""The bench where the compiled reference is not there: the reference arm says so in one line and
ends well, and our own arm goes without the CPU baseline."""
import json
import types

import bench
from oracle import ref


def test_reference_arm_says_that_it_is_unavailable(monkeypatch, capsys, tmp_path):
    monkeypatch.setattr(ref, "REF_SO", str(tmp_path / "liboref.so"))
    monkeypatch.delenv("RANK", raising=False)
    args = types.SimpleNamespace(workload=bench.DEFAULT_WORKLOAD, steps=1, warmup=3, gpus=1)
    assert bench.run_reference(args) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "liboref.so" in line["unavailable"]


def test_our_arm_goes_without_the_baseline(monkeypatch, tmp_path):
    monkeypatch.setattr(ref, "REF_SO", str(tmp_path / "liboref.so"))
    seen = []

    class Stop(Exception):
        pass

    def ours(args):
        seen.append(args.no_cpu_baseline)
        raise Stop

    monkeypatch.setattr(bench, "Ours", ours)
    for given in (False, True):
        try:
            bench.run_ours(types.SimpleNamespace(no_cpu_baseline=given))
        except Stop:
            pass
    assert seen == [True, True]
    (tmp_path / "liboref.so").touch()
    try:
        bench.run_ours(types.SimpleNamespace(no_cpu_baseline=False))
    except Stop:
        pass
    assert seen[-1] is False
