"""Device memory of the chip-resident and streaming solves: a handle that fits
without their buffers is made without them, and solves."""
import numpy as np
import pytest

from flursys_b200 import _abi
from flursys_b200.solver import _Handle

from .test_gpu_cavity2d import cfg2d

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


def _footprint(cfg):
    before = _free()
    h = _Handle(cfg)
    used = before - _free()
    h.step(1)
    h.close()
    return used


def _pcg2d(oracle):
    c = cfg2d(oracle, 4000, 148, dt=1e-6, precision=_abi.PRECISION_MIXED)
    c.stop_rule, c.pressure_rtol, c.pressure_max_iters = _abi.STOP_REL_L2, 1e-8, 20
    return c, "FLURSYS_2D_RESIDENT", _abi.FIELD_PRESSURE


def _sor3d(oracle):
    c = oracle.default_config(3)
    c.nx, c.ny, c.nz = 100, 62, 148
    c.pressure_max_iters, c.pressure_tolerance = 20, 1e-300
    return c, "FLURSYS_SOR_RESIDENT", _abi.FIELD_PRESSURE


@pytest.mark.parametrize("case", [_pcg2d, _sor3d])
def test_no_room_for_the_resident_records(oracle, monkeypatch, case):
    import torch
    cfg, env, field = case(oracle)
    monkeypatch.setenv(env, "0")
    _footprint(cfg)  # the modules load
    plain = _footprint(cfg)
    h = _Handle(cfg)
    h.step(1)
    ref = h.download(field)
    h.close()
    monkeypatch.setenv(env, "1")
    _footprint(cfg)
    resident = _footprint(cfg)
    assert resident - plain >= 24 * MB  # the records, in one allocation
    torch.cuda.empty_cache()
    room = plain + 10 * MB
    filler = torch.empty(_free() - room, dtype=torch.uint8, device="cuda")
    try:
        assert plain + 4 * MB <= _free() <= resident - 4 * MB
        h = _Handle(cfg)
        h.step(1)
        p = h.download(field)
        h.close()
    finally:  # the other tests need the memory
        del filler
        torch.cuda.empty_cache()
    assert np.array_equal(p, ref)  # the streaming kernel's result


@pytest.mark.parametrize("form,precision,vectors", [
    ("stream", _abi.PRECISION_F64, 1 * 8),    # the graph holds r, two d and q; this form two r, two d and the increment
    ("stream", _abi.PRECISION_MIXED, 0),      # the graph has the increment too
    ("grid", _abi.PRECISION_MIXED, -5 * 4),   # rows: all on the chip
])
def test_a_form_with_its_own_vectors_does_not_hold_the_graphs(oracle, monkeypatch, form, precision, vectors):
    from .test_gpu_cavity3d import cfg3d
    shape = (160, 160, 160) if form == "stream" else (128, 128, 128)
    cfg = cfg3d(oracle, *shape, precision=precision)
    cfg.pressure_max_iters = 20
    used = {}
    for env in ("0", form):
        monkeypatch.setenv("FLURSYS_PCG_RESIDENT", env)
        _footprint(cfg)
        used[env] = _footprint(cfg)
    # records, faces and the rounding of allocations to 2 MB: a few MB
    assert used[form] - used["0"] <= vectors * np.prod(shape) + 16 * MB
