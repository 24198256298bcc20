"""An engine and a batch run on streams of their own, which do not wait for the default stream:
what their kernels read is uploaded on the same stream (the calls' copies and the streams they
ran on, as the profiler reports them)."""
import numpy as np
import pytest

from aerosim_b200 import LBMBatch, cases, sgs

pytestmark = pytest.mark.gpu


def _streams(call):
    """Streams of the kernels and of the host-to-device copies and memsets of call()."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1).cuda()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    kernels, uploads = {}, {}
    for e in p.profiler.kineto_results.events():
        if e.device_type() != torch.autograd.DeviceType.CUDA:
            continue
        if e.name().startswith(("Memcpy HtoD", "Memset")):
            uploads.setdefault(e.device_resource_id(), []).append(e.name())
        elif not e.name().startswith("Mem"):
            kernels.setdefault(e.device_resource_id(), []).append(e.name())
    if not kernels and not uploads:
        pytest.skip("the profiler sees no device activity on this machine")
    return kernels, uploads


def _engine(cls, case):
    e = cls(0)
    e.voxelize(case.mesh, None, case.tunnel, {"nx": case.nx, "ny": case.ny, "nz": case.nz},
               {"uInletLattice": case.u_inlet, "nuLattice": case.nu, "smagorinskyCs": case.cs, "precision": "f32"})
    return e


def test_uploads_of_an_engine_are_on_its_stream(gpu_engine_cls):
    case = cases.sphere_64x32x32()
    e = _engine(gpu_engine_cls, case)
    grid, other = e.read_voxel_grid(), gpu_engine_cls(0)
    assert grid.boundaryCellCount > 0
    cfg = {k: e.config[k] for k in ("uInletLattice", "nuLattice", "smagorinskyCs", "precision", "tunnel")}
    for call in (lambda: other.set_voxel_grid(grid, cfg), lambda: (other.set_sgs_mlp(sgs.init_params(1)), other.step(2))):
        kernels, uploads = _streams(call)
        assert len(kernels) == 1 and uploads, (kernels, uploads)
        assert set(uploads) == set(kernels), (kernels, uploads)
    e.close(), other.close()


def test_uploads_of_a_batch_are_on_streams_with_kernels(gpu_engine_cls):
    case = cases.sphere_64x32x32()
    es = [_engine(gpu_engine_cls, case) for _ in range(2)]
    made = []

    def call():
        made.append(LBMBatch(es))
        made[0].set_tuning(2, 1, 1, 512)
        made[0].step(2)

    kernels, uploads = _streams(call)
    assert len(kernels) == 3 and uploads  # two engines' resets, the batch's steps
    assert set(uploads) <= set(kernels), (kernels, uploads)
    made[0].close()
    for e in es:
        e.close()
