"""The similarity operators on every form of the search image they take: uint8
and uint16 pixels, host and device memory, rows longer than the image; and on
more poses than the GPU has SMs.  Scores and gradients against the FP64
restatement within its bounds (2e-6; 1e-4 + 1e-3 relative); refinements bit for
bit the same for all forms of one image, by one block a pose or by the cluster of
four that rows a multiple of 256 bytes apart take (templates of 12288 samples or
more)."""
import math

import numpy as np
import pytest

import oracle_lib
from mvkit_gb300 import workloads as W
from test_gpu_adjoint import ncc64, poses_near_truth

pytestmark = pytest.mark.gpu
A = math.radians(10)


def image_form(mg, image, place, pad):
    """`image` as the operators take it: rows `pad` pixels longer than it."""
    h, w = image.shape
    store = np.full((h, w + pad), 77, image.dtype)
    store[:, :w] = image
    if place == "host":
        return store[:, :w]
    dev = mg.DeviceImage(store)
    dev.shape = (h, w)
    return dev


@pytest.mark.parametrize("place, pad", [("host", 13), ("device", 0), ("device", 13)])
@pytest.mark.parametrize("maxval", [255, 4095])
def test_forms_of_the_image(maxval, place, pad):
    import mvkit_gb300 as mg

    wl = W.make_workload(31, 307, 391, 53, 2, angle_range=(-A, A), maxval=maxval,
                         noise_sigma=3 if maxval == 255 else 20)
    model = mg.create_ncc_model(wl.template, 2, -A, 2 * A, "auto", "use_polarity")
    om = oracle_lib.oracle().create(wl.template, levels=2, angle_start=-A, angle_extent=2 * A)
    p = om.patch(-1, 0)
    dr, dc, w = p["rows"] - p["origin_row"], p["cols"] - p["origin_column"], p["weights"]
    image = image_form(mg, wl.image, place, pad)
    poses = poses_near_truth(wl, 3, per=2)
    poses = np.concatenate([poses, [[1.0, 2.0, 0.0, 1.0], [305.0, 389.0, 0.1, 1.0]]])  # samples outside
    score, grad = mg.ncc_score_gradient(image, model, poses)
    for k, pose in enumerate(poses):
        s64, g64 = ncc64(wl.image, dr, dc, w, pose)
        assert score[k] == s64 or abs(score[k] - s64) <= 2e-6
        assert np.all(np.abs(grad[k] - g64) <= 1e-4 + 1e-3 * np.abs(g64))
    want = mg.ncc_refine_similarity(np.ascontiguousarray(wl.image), model, poses, iterations=12)
    got = mg.ncc_refine_similarity(image, model, poses, iterations=12)
    assert np.all(want[1][:4] > score[:4])
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("maxval", [255, 4095])
def test_more_poses_than_sms(maxval):
    import mvkit_gb300 as mg

    wl = W.make_workload(32, 420, 500, 113, 2, angle_range=(-A, A), maxval=maxval,
                         noise_sigma=3 if maxval == 255 else 20)
    model = mg.create_ncc_model(wl.template, 2, -A, 2 * A, "auto", "use_polarity")
    poses = poses_near_truth(wl, 9, per=3)
    alone = mg.ncc_refine_similarity(wl.image, model, poses, iterations=12)
    team = mg.ncc_refine_similarity(image_form(mg, wl.image, "host", 512 - 500), model, poses, iterations=12)
    assert np.array_equal(team[0], alone[0]) and np.array_equal(team[1], alone[1])
    many = mg.ncc_refine_similarity(wl.image, model, np.tile(poses, (100, 1)), iterations=12)
    assert np.array_equal(many[0], np.tile(alone[0], (100, 1))) and np.array_equal(many[1], np.tile(alone[1], 100))
    s, g = mg.ncc_score_gradient(wl.image, model, poses)
    sm, gm = mg.ncc_score_gradient(wl.image, model, np.tile(poses, (100, 1)))
    assert np.array_equal(sm, np.tile(s, 100)) and np.array_equal(gm, np.tile(g, (100, 1)))
