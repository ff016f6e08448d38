"""The benchmark's reference arm runs the reference's own code or nothing."""
import json


def test_reference_arm_without_the_reference_says_so(monkeypatch, tmp_path, capsys):
    import bench

    class A:
        n, nt, groups, steps, warmup, gpus = 201, 1501, 4, 1, 0, 1

    def no_stand_in(*args):
        raise AssertionError("another implementation was timed in the reference's place")
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))
    monkeypatch.setattr(bench, "ref_inputs", no_stand_in)
    monkeypatch.setattr(bench, "reference_sample", no_stand_in)
    bench.run_reference(A(), rank=0)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "afdcfun" in line["unavailable"]


def test_reference_build_is_found(monkeypatch, tmp_path):
    import bench
    (tmp_path / "oracle" / "_ref").mkdir(parents=True)
    (tmp_path / "oracle" / "_ref" / "afdcfun.py").write_text("")
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))
    assert bench.reference_built()
