"""The source hash that ties a profile to a build covers every source folder."""
import os
import shutil

import bench


def test_source_sha_covers_every_folder(tmp_path, monkeypatch):
    csrc = os.path.join(bench.ROOT, "profess_b200", "csrc")
    copy = tmp_path / "profess_b200" / "csrc"
    shutil.copytree(csrc, copy)
    built = bench.source_sha()
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))
    assert bench.source_sha() == built
    for d, _, files in os.walk(copy):
        for name in files:
            if not name.endswith((".cu", ".cuh")):
                continue
            path = os.path.join(d, name)
            text = open(path).read()
            with open(path, "w") as fh:
                fh.write(text + "\n")
            assert bench.source_sha() != built, path
            with open(path, "w") as fh:
                fh.write(text)
    assert bench.source_sha() == built
