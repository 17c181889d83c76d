"""The tuner's on-disk cache of launch shapes, on the CPU with a plan that
only records what is asked of it."""

import json

import pytest
import torch

from tmol_b200 import tune


class FakePlan:
    NAME = "LJ/LK"
    device, dtype, n_poses, max_n_blocks = "cuda:0", torch.float32, 2, 10

    def __init__(self):
        self.block_sizes = (torch.zeros(2, 10, dtype=torch.int32), torch.tensor([20], dtype=torch.int32))
        self.shapes = []

    def set_launch(self, *shape):
        self.shapes.append(shape)

    def balance(self, run):
        pass

    def profile(self, on):
        pass

    def profile_read(self):
        return float(len(set(self.shapes))), 1


@pytest.fixture
def cache_file(tmp_path, monkeypatch):
    monkeypatch.setenv("TMOL_B200_TUNE_CACHE", str(tmp_path / "launch.json"))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device: "NVIDIA B200")
    return tmp_path / "launch.json"


def test_shapes_of_other_kernels_are_not_taken(cache_file):
    """A file from before the kernels' launch shapes changed (12 slots, at
    most 16 warps) does not decide for the ones that are there."""
    plan = FakePlan()
    old = "NVIDIA B200|LJ/LK|torch.float32|P=2|B=10|blocks/pose=10|atoms/block=20|sizes%=0,0,100,0,0"
    assert tune.signature(plan).endswith(old.split("|", 1)[1])
    cache_file.write_text(json.dumps({old: {"shape": [1, 16, 1, 64, 12], "ms": 1.0}}))
    shape, _ = tune.autotune(plan, lambda: None)
    shapes = list(tune.launch_shapes(tune.DEFAULT_GRID))
    assert shape in shapes and set(plan.shapes) == set(shapes)
    assert json.loads(cache_file.read_text())[old]["shape"] == [1, 16, 1, 64, 12]


def test_tuned_shape_is_taken_again(cache_file):
    first, _ = tune.autotune(FakePlan(), lambda: None)
    plan = FakePlan()
    assert tune.autotune(plan, lambda: None)[0] == first
    assert plan.shapes == [first]
