"""The benchmark's result line: one line on stdout, whole, with the tables beside it."""
import json


def test_result_line_is_short_and_the_tables_are_not_lost(capsys):
    import bench
    row = {"kind": "conv3", "c": 256, "dtype": "fp16", "voxels_in": 500000, "ms": 0.11091199964284897, "useful_tflops": 590.8828639915828}
    line = {"metric": bench.METRIC, "value": 284812345.678901, "unit": bench.UNIT, "ms_per_step": 4.213456789012345,
            "roofline": {"frac": 0.2876543210987, "by_shape": [row] * 8}, "kmap": [row] * 16, "layers": [row] * 24, "config5": None}
    bench.print_result(line)
    out, err = capsys.readouterr()
    (only,) = out.splitlines()
    got = json.loads(only)
    assert len(only) < 1000 and got["value"] == 284812000.0 and got["ms_per_step"] == 4.21346 and got["roofline"] == {"frac": 0.287654}
    tables = {}
    for text in err.splitlines():
        tables.update(json.loads(text))
    assert {k: len(v) for k, v in tables.items()} == {"kmap": 16, "layers": 24, "roofline.by_shape": 8}
