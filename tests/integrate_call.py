"""The batched integrator called on a prepared batch's device arrays, so that
tests can alter them (the ray tables among them) between the stages."""
import ctypes as C

from xpsi_gb300 import _native as N


def batch_data(ev, B):
    """xgpu_integrate_batch's data for the buffers of BatchEvaluator.upload()."""
    p = lambda x: x.data_ptr()
    row = B["row"]
    d = N.IntegrateBatchData()
    d.row_mesh = p(B["row_mesh"])
    d.radius, d.u, d.cos_gamma = p(row["radius"]), p(row["u"]), p(row["cos_gamma"])
    d.theta0, d.maxDeflection = p(row["theta0"]), p(B["maxDefl"])
    d.deflection, d.cos_alpha, d.lag = p(B["defl"]), p(B["ca"]), p(B["lag"])
    d.cellArea, d.phi, d.params, d.n_params = p(B["cellArea"]), p(B["phi"]), p(B["params"]), 2
    d.radiates = p(B["radiates"])
    d.energies, d.leaves, d.phases = p(ev.energies), p(ev.leaves), p(ev.phases)
    if ev.atmos is not None:
        d.atmos = ev.atmos
    d.flux, d.mesh_status = p(B["flux"]), p(B["mesh_status"])
    if "correction" in B:
        d.correction, d.n_correction = p(B["correction"]), 2
    return d


def integrate(ev, B):
    """Fluxes [members, N_E, N_P] and the members' statuses."""
    torch = ev.torch
    P, d = B["P"], batch_data(ev, B)
    f = N.lib().xgpu_integrate_batch_mixed if ev.precision == "mixed" else \
        N.lib().xgpu_integrate_batch
    N.check(f(P.V * P.H, P.meshes, P.n_rows, ev.N_R, len(ev.model.energies), ev.N_L, ev.N_L,
              C.byref(d), int(ev.target_ctas), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return B["flux"].cpu().numpy(), B["mesh_status"].cpu().numpy()


def integrate_scratch(ev, B, limit_bytes=0):
    """integrate() with a bound on the call's scratch: fluxes, statuses, what
    the call reports, and the parallels that found no geometry records."""
    torch = ev.torch
    P, d = B["P"], batch_data(ev, B)
    count = torch.full((1,), -1, dtype=torch.int64, device=ev.dev)
    s = N.IntegrateScratch(limit_bytes, count.data_ptr())
    N.check(N.lib().xgpu_integrate_batch_scratch(
        P.V * P.H, P.meshes, P.n_rows, ev.N_R, len(ev.model.energies), ev.N_L, ev.N_L, C.byref(d),
        int(ev.target_ctas), int(ev.precision == "mixed"), C.byref(s),
        torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return B["flux"].cpu().numpy(), B["mesh_status"].cpu().numpy(), s, int(count.item())
