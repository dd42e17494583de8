"""The kernels that a batch run says it launches per step, against a profile of one step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n,kind,layout,count,tuning", [
    (16, "GEN_HEIGHTMAP", 0, 1024, {}), (16, "GEN_HEIGHTMAP", 0, 5000, {}), (16, "GEN_HEIGHTMAP", 1, 5000, {}),
    (8, "GEN_HEIGHTMAP", 0, 7000, {}), (32, "GEN_DENSITY", 0, 100, {}), (32, "GEN_BERNOULLI", 0, 40, {}),
    (16, "GEN_HEIGHTMAP", 0, 1000, {"ctas_per_sm": 2}), (16, "GEN_HEIGHTMAP", 0, 5000, {"slab_chunks": 2000}),
    (16, "GEN_DENSITY", 0, 500, {"halo_staging": 1}), (16, "GEN_HEIGHTMAP", 0, 500, {"schedule": 0})])
def test_kernels_per_step(vox, graph, n, kind, layout, count, tuning):
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile

    from voxgpu.batch import BatchRun
    cfg = vox.make_config(chunk_size=n, kind=getattr(vox, kind), layout=layout, octaves=2, frequency=1 / 90,
                          y_ref=0.0, y_scale=1 / 64)
    ctx = vox.Context(cfg, stream=torch.cuda.current_stream().cuda_stream or 1)
    t = ctx.tuning()
    ctx.set_tuning(t.threads, t.stage_faces, tuning.get("ctas_per_sm", 0), tuning.get("schedule", t.schedule),
                   tuning.get("slab_chunks", 0), tuning.get("halo_staging", 0))
    side = int(np.ceil(np.sqrt(count)))
    coords = [(i % side, 0, i // side) for i in range(count)]
    run = BatchRun(ctx, coords, None if kind == "GEN_BERNOULLI" else [15] * count, graph=graph)
    run.launch()
    ctx.sync()
    for _ in range(2):  # a process's first profile may come back empty
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            run.launch()
            ctx.sync()
        kernels = [e for e in prof.events() if "k_" in e.name and "vox::" in e.name]
        if kernels:
            break
    if not kernels:
        pytest.skip("no kernel activity from the profiler")
    assert run.kernels_per_step == len(kernels), [e.name for e in kernels]
    run.close()
    ctx.close()
