"""bench.py's result line: one line of JSON on stdout, the long side measurements not
in it."""
import json


def test_result_line_is_short_and_alone_on_stdout(capsys):
    import bench
    side = {"config %d" % i: "x" * 100 for i in range(200)}
    bench.emit({"metric": "m", "value": 1.5, "gpu_launches": 3}, side)
    got = capsys.readouterr()
    lines = got.out.splitlines()
    assert len(lines) == 1 and len(lines[0]) < 4000
    assert json.loads(lines[0]) == {"metric": "m", "value": 1.5, "gpu_launches": 3}
    assert json.loads(got.err) == {"other_configs": side}
