// Fault_qd::d_dt for one fault node (its four lanes together, see
// fault_dev.cuh), shared by the linear-elastic, response-mode and power-law
// drivers.
#pragma once
#include "fault_dev.cuh"

namespace scy {

// A node's parameters, laid out by the host: a launch requests them ahead of
// what it waits for (the kernel before, the node's stress).  In turn on one
// GPU eight response steps at 401 nodes took 592 us so and 640 with the loads
// in the update, four solve steps at 101 x 101 775 and 787 (600 to 617 and 760
// to 780 over several GPUs).
struct FaultNode {
  double prestress, a, b, sN, Dc, eta, locked;
};
__device__ __forceinline__ FaultNode fault_node_load(const FaultParams& fp, int iz) {
  return FaultNode{fp.prestress[iz], fp.a[iz], fp.b[iz], fp.sN[iz], fp.Dc[iz], fp.eta[iz], fp.locked[iz]};
}

// Fault_qd::d_dt for one node given its quasi-static shear stress from the
// body and its state psi (fault.cpp:861-918): prestress, bracketed Newton,
// state law, tauP, strength.  Lane 0 of the four stores.
__device__ __forceinline__ void fault_node_update(int iz, double tau_body, const FaultParams& fp, const FaultNode& n,
                                                  double psi, double* __restrict__ f, double* __restrict__ slipVel,
                                                  double* __restrict__ tauQSP, double* __restrict__ tauP,
                                                  double* __restrict__ strength, unsigned* flags,
                                                  unsigned long long* its_total) {
  const bool out = (threadIdx.x & 3) == 0;
  const double tq = tau_body + n.prestress;
  const double a = n.a, sN = n.sN, eta = n.eta;
  const double E = exp(psi / a), V0 = slipVel[iz];
  __syncwarp(node_lanes());  // every lane has V0 before lane 0 overwrites it
  double V;
  const double lk = n.locked;
  if (lk > 0.5) {
    V = 0.0;
  } else if (lk < -0.5) {
    V = fp.vL;
  } else {
    double left = 0.0, right = tq / eta;
    if (isnan(right)) {
      if (out) atomicOr(flags, (unsigned)FAULT_NONFINITE);
      V = V0;
    } else if (fabs(left - right) < 1e-14) {
      V = left;
    } else {
      int its = 0;
      bool ok = true;
      const ResidQD R{tq, eta, sN, E, a, fp.v0, fp.jacobian};
      V = bracketed_newton_f(R, left, right, V0, fp.root_tol, fp.max_its, &its, &ok);
      if (out) {
        atomicAdd(its_total, (unsigned long long)its);
        if (!ok) atomicOr(flags, (unsigned)FAULT_ROOT_NOCONV);
      }
    }
  }
  const double S = asinh((0.5 * V / fp.v0) * E);  // of the strength and, in magnitude, of the slip law
  double dpsi;
  if (fp.state_law == 0)
    dpsi = aging_law_psi(psi, V, n.b, fp.f0, fp.v0, n.Dc);
  else if (fp.state_law == 1)
    dpsi = slip_law_of_asinh(fabs(S), V, a, n.b, fp.f0, fp.v0, n.Dc);
  else if (fp.state_law == 3) {
    // flashHeating_psi_Vec (fault.cpp:2199-2243): Vw from the fault's temperature
    const double vw = flash_heating_vw(fp.Tf[iz], fp.rc_f[iz], fp.k_f[iz], fp.fl_D, fp.Tw[iz], fp.fl_tau_c);
    if (out) fp.Vw[iz] = vw;
    dpsi = flash_heating_psi(psi, V, vw, fp.fl_fw, n.Dc, a, n.b, fp.f0, fp.v0);
  } else
    dpsi = 0.0;
  if (!out) return;
  if (!isfinite(dpsi) || !isfinite(V)) atomicOr(flags, (unsigned)FAULT_NONFINITE);
  tauQSP[iz] = tq;
  slipVel[iz] = V;
  f[fp.psi_off + iz] = dpsi;
  f[fp.slip_off + iz] = V;
  tauP[iz] = tq - eta * V;
  strength[iz] = a * sN * S;
}

}  // namespace scy
