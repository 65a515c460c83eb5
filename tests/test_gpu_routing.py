"""At-floor routing census on the B200: bit-identical to the reference.

Every golden mask goes through route_at_floor_mask on the device and must
give the reference's census bytes and planes; seeded random masks (ragged
sizes, single rows and columns, perimeter rings, full-frame size) must match
the oracle; each device primitive is checked against its oracle restatement.
"""

from __future__ import annotations

import ctypes
import hashlib
import json
import os

import numpy as np
import pytest

import route_cases
from fauxice_b200 import _lib, routing
from oracle import routing_oracle as ro

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def sha(data: bytes) -> str:
    return hashlib.sha256(data).hexdigest()


@pytest.fixture(scope="module")
def route_golden():
    with open(os.path.join(HERE, "golden", "routing_golden.json")) as handle:
        return json.load(handle)["cases"]


@pytest.mark.parametrize("name", list(route_cases.CASES))
def test_device_census_matches_reference(name, route_golden):
    expected = route_golden[name]
    mask = route_cases.mask(name)
    policy = routing.RoutingPolicy(**route_cases.policy_kwargs(name))
    if "error" in expected:
        with pytest.raises(routing.NoHealthyContextError) as raised:
            routing.route_at_floor_mask(mask, policy)
        assert raised.value.image_shape == mask.shape
        assert raised.value.finite_radius_sentinel == max(mask.shape)
        return
    result = routing.route_at_floor_mask(mask, policy)
    payload = routing.serialize_routing_json(result)
    if "json" in expected and sha(payload) != expected["json_sha256"]:
        assert payload.decode("utf-8") == expected["json"]
    assert sha(payload) == expected["json_sha256"]
    assert sha(result.provisional_labels.tobytes()) == expected["provisional_labels_sha256"]
    assert sha(result.synthesis_mask.tobytes()) == expected["synthesis_mask_sha256"]
    assert sha(result.final_labels.tobytes()) == expected["final_labels_sha256"]
    for plane in (result.provisional_labels, result.synthesis_mask, result.final_labels):
        assert not plane.flags.writeable


def test_device_tensor_input_matches_host_input():
    import torch

    mask = route_cases.mask("perimeter_ring_80x100")
    host = routing.serialize_routing_json(routing.route_at_floor_mask(mask))
    device = routing.serialize_routing_json(
        routing.route_at_floor_mask(torch.from_numpy(mask).to("cuda")))
    assert host == device


def _random_mask(seed: int) -> tuple[np.ndarray, dict]:
    rng = np.random.default_rng(seed)
    kind = seed % 5
    if kind == 0:
        h, w = int(rng.integers(1, 4)), int(rng.integers(1, 700))
        m = rng.random((h, w)) < rng.uniform(0.1, 0.8)
    elif kind == 1:
        h, w = int(rng.integers(1, 700)), int(rng.integers(1, 4))
        m = rng.random((h, w)) < rng.uniform(0.1, 0.8)
    elif kind == 2:
        h, w = int(rng.integers(33, 400)), int(rng.integers(33, 400))
        m = route_cases.perimeter_ring(seed, h, w, thickness=int(rng.integers(1, 5)))
    elif kind == 3:
        h, w = int(rng.integers(40, 700)), int(rng.integers(40, 700))
        m = route_cases.dust(seed, h, w, count=int(rng.integers(1, 80)), rmax=20)
    else:
        h, w = int(rng.integers(20, 500)), int(rng.integers(20, 500))
        m = rng.random((h, w)) < rng.uniform(0.2, 0.6)
    policy = {"min_area": int(rng.integers(1, 500)), "min_radius": int(rng.integers(1, 8)),
              "margin": int(rng.integers(0, 12)),
              "max_synth_fraction": float(rng.choice([0.0, 0.02, 0.25, 1.0]))}
    if m.all():
        m[0, 0] = False
    return m, policy


@pytest.mark.parametrize("seed", range(40))
def test_device_census_matches_oracle_on_random_masks(seed):
    mask, policy = _random_mask(seed)
    doc, prov, synth, final = ro.route(mask, **policy)
    result = routing.route_at_floor_mask(mask, routing.RoutingPolicy(**policy))
    assert routing.serialize_routing_json(result) == ro.serialize(doc)
    assert np.array_equal(result.provisional_labels, prov)
    assert np.array_equal(result.synthesis_mask, synth)
    assert np.array_equal(result.final_labels, final)


def test_full_frame_dust_matches_oracle():
    """A full-frame mask (4000 x 5700, 22.8 MP) with thousands of regions."""

    mask = route_cases.dust(21, 4000, 5700, count=6000, rmax=24)
    doc, prov, synth, final = ro.route(mask)
    result = routing.route_at_floor_mask(mask)
    assert routing.serialize_routing_json(result) == ro.serialize(doc)
    assert np.array_equal(result.final_labels, final)
    assert np.array_equal(result.provisional_labels, prov)


# --- primitives -------------------------------------------------------------


def _dev():
    return routing._Device()


@pytest.mark.parametrize("shape, density", [((1, 1), 1.0), ((1, 513), 0.5), ((517, 1), 0.5),
                                            ((255, 257), 0.3), ((500, 700), 0.55),
                                            ((1024, 768), 0.7), ((300, 300), 0.0)])
def test_label8_matches_oracle(shape, density):
    import torch

    rng = np.random.default_rng(shape[0] * 7 + shape[1])
    mask = rng.random(shape) < density
    dev = _dev()
    labels, count = dev.label8(torch.from_numpy(mask.view(np.uint8)).cuda(), *shape)
    expected, expected_count = ro.label8(mask)
    assert count == expected_count
    assert np.array_equal(labels.cpu().numpy(), expected)


@pytest.mark.parametrize("shape, density", [((1, 300), 0.8), ((300, 1), 0.8), ((257, 129), 0.9),
                                            ((600, 450), 0.97), ((64, 64), 0.5)])
def test_chessboard_distance_matches_oracle(shape, density):
    import torch

    rng = np.random.default_rng(shape[0] + 3 * shape[1])
    mask = rng.random(shape) < density
    mask[rng.integers(0, shape[0]), rng.integers(0, shape[1])] = False
    dist = _dev().distance(torch.from_numpy(mask.view(np.uint8)).cuda(), *shape)
    assert np.array_equal(dist.cpu().numpy(), ro.chessboard_distance(mask))


@pytest.mark.parametrize("radius", [0, 1, 3, 17, 5000])
def test_square_dilation_matches_oracle(radius):
    import torch

    rng = np.random.default_rng(radius)
    mask = rng.random((211, 389)) < 0.002
    out = _dev().dilate(torch.from_numpy(mask.view(np.uint8)).cuda(), 211, 389, radius)
    assert np.array_equal(out.cpu().numpy().view(np.bool_), ro.dilate_square(mask, radius))


def test_primitives_reject_bad_arguments():
    lib = _lib.load()
    count = ctypes.c_int64()
    assert lib.fx_label8(None, 4, 4, None, None, None, None, ctypes.byref(count), None) == 1
    assert lib.fx_tile_extract(ctypes.c_void_p(16), 4, 4, 2, 2, 3, 3, 1, ctypes.c_void_p(16),
                               None) == 1  # tile outside the plane: rejected before launch


@pytest.mark.parametrize("shape", [(65, 31), (64, 32), (130, 33), (200, 257), (3, 640), (640, 3)])
@pytest.mark.parametrize("fill", ["stripes", "full", "corner"])
def test_deep_and_word_edge_shapes_match_oracle(shape, fill):
    """Words that end a row, tiles that end the frame, components that cross
    word boundaries, and distances on both sides of the bit plane's reach."""

    import torch

    h, w = shape
    mask = np.ones(shape, bool)
    if fill == "stripes":
        mask[:, 31::33] = False
        mask[::7, ::5] = False
    elif fill == "full":
        mask[h // 2, w // 2] = False
    else:
        mask[0, 0] = False
    dev = _dev()
    m = torch.from_numpy(mask.view(np.uint8)).cuda()
    labels, count = dev.label8(m, h, w)
    expected, expected_count = ro.label8(mask)
    assert count == expected_count
    assert np.array_equal(labels.cpu().numpy(), expected)
    dist = dev.distance(m, h, w)
    assert np.array_equal(dist.cpu().numpy(), ro.chessboard_distance(mask))
    areas, boxes, maxima = dev.stats(labels, dist, h, w, count)
    d = dist.cpu().numpy()
    for k in range(count):
        ys, xs = np.nonzero(expected == k + 1)
        assert areas[k] == ys.size and maxima[k] == d[ys, xs].max()
        assert list(boxes[k]) == [ys.min(), xs.min(), ys.max() + 1, xs.max() + 1]
    counts = dev.count_where(labels, (dist > 1).int(), count)
    assert [counts[k + 1] for k in range(count)] == [
        int(((expected == k + 1) & (d > 1)).sum()) for k in range(count)]


@pytest.mark.parametrize("radius", [1, 15, 16, 30, 31, 32, 40])
@pytest.mark.parametrize("shape", [(1, 700), (700, 1), (64, 256), (65, 257), (130, 31)])
def test_dilation_tiles_match_oracle(shape, radius):
    import torch

    mask = np.random.default_rng(radius).random(shape) < 0.004
    mask[shape[0] // 2, shape[1] // 2] = True
    out = _dev().dilate(torch.from_numpy(mask.view(np.uint8)).cuda(), *shape, radius)
    assert np.array_equal(out.cpu().numpy().view(np.bool_), ro.dilate_square(mask, radius))


# rows of 16-row tiles on both sides of 65,535, the blocks of a grid's second axis, and of
# the 32-row tiles of the relaxation, which the gap of 300 rows reaches
@pytest.mark.parametrize("h, w", [(1048560, 1), (1048577, 1), (1048577, 40), (2097153, 1)])
def test_chessboard_distance_of_tall_masks(h, w):
    import torch

    rows = np.arange(h)
    background = np.concatenate([rows[:h - 400:50], rows[h - 101:]])  # whole rows
    mask = np.ones((h, w), np.uint8)
    mask[background] = 0
    after = np.searchsorted(background, rows)
    expected = np.minimum(np.abs(rows - background[np.minimum(after, len(background) - 1)]),
                          np.abs(rows - background[np.maximum(after - 1, 0)]))
    assert expected.max() >= 150
    dist = _dev().distance(torch.from_numpy(mask).cuda(), h, w).cpu().numpy()
    assert np.array_equal(dist, np.broadcast_to(expected[:, None], (h, w)))


def test_census_of_a_tall_mask_measures_its_regions():
    mask = np.zeros((1048577, 1), bool)
    mask[1000:1040] = mask[700000:700003] = mask[-90:-20] = True
    result = routing.route_at_floor_mask(mask)
    assert [(r.area, r.max_chessboard_radius) for r in result.provisional_regions] == [
        (40, 20), (3, 2), (70, 35)]


@pytest.mark.parametrize("offset", [0, 1, 1500])  # the output's start in the input plane
@pytest.mark.parametrize("radius", [1, 12, 31])
def test_dilation_in_place_matches_oracle(radius, offset):
    import torch

    h, w = 700, 1100
    mask = np.random.default_rng(radius).random((h, w)) < 0.001
    plane = torch.zeros(h * w + offset, dtype=torch.uint8, device="cuda")
    plane[:h * w] = torch.from_numpy(mask.view(np.uint8).ravel()).cuda()
    work = torch.empty(h * w, dtype=torch.uint8, device="cuda")
    at = plane.data_ptr()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert _lib.load().fx_dilate_square(ctypes.c_void_p(at), h, w, radius,
                                        ctypes.c_void_p(work.data_ptr()),
                                        ctypes.c_void_p(at + offset), stream) == 0
    out = plane[offset:].cpu().numpy().reshape(h, w)
    assert np.array_equal(out.view(np.bool_), ro.dilate_square(mask, radius))


@pytest.mark.parametrize("shape", [(300, 300), (701, 933), (97, 63)])
@pytest.mark.parametrize("kind", ["stripes", "checker", "noise"])
def test_many_links_a_word_match_oracle(shape, kind):
    import torch

    y, x = np.ogrid[:shape[0], :shape[1]]
    mask = {"stripes": (x % 2 == 0) & (y >= 0), "checker": (x + y) % 2 == 0,
            "noise": np.random.default_rng(shape[0]).random(shape) < 0.5}[kind]
    labels, count = _dev().label8(torch.from_numpy(mask.view(np.uint8)).cuda(), *shape)
    expected, expected_count = ro.label8(mask)
    assert count == expected_count
    assert np.array_equal(labels.cpu().numpy(), expected)
