"""The bench's records: when the captured DRAM traffic still counts, and what goes into the result line."""
import json
import shutil

import bench


def test_traffic_record_is_stale_once_a_source_that_decides_traffic_changes(tmp_path, monkeypatch):
    names = [p.rsplit("/", 1)[1] for p in bench.TRAFFIC_SOURCES]
    assert {"conv_tc_kernel.cuh", "conv_tc.cu"} <= set(names)
    copies = [str(tmp_path / n) for n in names]
    for src, dst in zip(bench.TRAFFIC_SOURCES, copies):
        shutil.copy(src, dst)
    monkeypatch.setattr(bench, "TRAFFIC_SOURCES", copies)
    record = tmp_path / "record.md"
    record.write_text("dram_bytes_per_launch = 1e6\nconv_tc_sha256 = %s\n" % bench.traffic_sources_sha256())
    monkeypatch.setattr(bench, "TRAFFIC_RECORD", str(record))
    assert bench.ncu_traffic_record()[:2] == (1e6, False)
    for path in copies:
        before = open(path).read()
        open(path, "a").write("\n")
        assert bench.ncu_traffic_record()[:2] == (None, True)
        open(path, "w").write(before)
    assert bench.ncu_traffic_record()[:2] == (1e6, False)


def test_the_result_is_one_line_without_the_networks_tables(capsys):
    rows = [{"name": "s5b4.conv2", "shape": "3x3 512->512 @19", "outputs": "residual+f32+i8", "us": 27.11, "frac": 0.2993}] * 72
    bench.emit({"metric": "m", "value": 1 / 3, "n": 123456789, "layers": rows[:5], "resnet50": {"ms": 1.0, "layers": rows}, "cspdarknet53": {"ms": 2.0, "layers": rows}})
    out, err = capsys.readouterr()
    line = json.loads(out)
    assert out.count("\n") == 1 and line["value"] == 0.3333333 and line["n"] == 123456789 and line["resnet50"] == {"ms": 1.0} and line["cspdarknet53"] == {"ms": 2.0} and len(line["layers"]) == 5
    tables = dict((l.split(" layers ", 1)[0], json.loads(l.split(" layers ", 1)[1])) for l in err.splitlines())
    assert tables == {"resnet50": rows, "cspdarknet53": rows}
