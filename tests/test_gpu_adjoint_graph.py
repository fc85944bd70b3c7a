"""A captured demigration replayed after set_model follows the new model, as the eager call does."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import migration, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,kernel", [(2, "demigrate_rows"), (16, "demigrate_cluster")])
def test_replayed_demigration_follows_set_model(ns, kernel):
    import torch
    dev = torch.device("cuda")
    w = synthetic.plain_medium(nx=256, nz=8, nf=3, ns=ns)
    om, vel = torch.from_numpy(w.omega).to(dev), torch.from_numpy(np.ascontiguousarray(w.velocity)).to(dev)
    tab = torch.from_numpy(w.table).to(dev)
    other = tab * 0.5j  # another operator: spectra differ by (0.5j)^nz
    wave = torch.from_numpy(w.wave).to(dev)
    m = torch.randn((w.nz, w.nx), generator=torch.Generator("cuda").manual_seed(3), device=dev)
    plan = migration.Plan.for_workload(w, wide=True)  # a migration kernel that does not use the row-split table
    out, eager = torch.zeros_like(wave), torch.zeros_like(wave)
    plan.set_model(om, vel, w.dk, tab)
    plan.demigrate(m, wave, out)
    assert plan.describe_demigration()["kernel"] == kernel
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.demigrate(m, wave, out)
    plan.set_model(om, vel, w.dk, other)
    graph.replay()
    plan.demigrate(m, wave, eager)
    torch.cuda.synchronize()
    assert float(eager.abs().max()) > 0
    np.testing.assert_array_equal(out.cpu().numpy(), eager.cpu().numpy())
    del graph
    plan.close()
