"""bench.py's DRAM traffic comes from a committed capture, and only from one of the kernels it times."""
import json

import bench


def test_traffic_of_other_device_code_is_not_reported(tmp_path):
    profile = {"kernel": "k_search", "dram_bytes_per_key": 1751.4}
    path = tmp_path / "k_search_dram.json"
    for digest, want in ((None, None), ("0" * 64, None), (bench.device_code_digest(), 1751.4)):
        path.write_text(json.dumps(profile if digest is None else dict(profile, device_code=digest)))
        assert bench.traffic_per_key("secure", str(tmp_path)) == want
    assert bench.traffic_per_key("incremental", str(tmp_path)) is None
