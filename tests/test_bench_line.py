"""The bench's records: when the captured DRAM traffic still counts."""
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
