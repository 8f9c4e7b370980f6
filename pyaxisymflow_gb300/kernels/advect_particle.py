"""Vorticity advection by remeshed particles (kernels/advect_particle.py:5-68)
on the GPU: particles on the axis-mirrored (2 nr, nz) domain move by u dt,
their vorticity is interpolated back onto the mesh with the MP4 kernel, and
the particles are reset to the mesh. Same arguments and in-place semantics
as the reference; float64 CUDA tensors."""
import torch

from .. import _native as N
from ..core.particles_to_mesh import _check, _scratch


def _advect(z_particles, r_particles, vort_particles, vorticity, Z_double, R_double, grid_size_r,
            u_z, u_r, dx, dt, periodic):
    nr = int(grid_size_r)
    nz = vorticity.shape[1]
    N.require(z_particles, r_particles, vort_particles, Z_double, R_double, shape=(2 * nr, nz),
              dtype=torch.float64,
              names=("z_particles", "r_particles", "vort_particles", "Z_double", "R_double"))
    N.require(vorticity, u_z, u_r, shape=(nr, nz), dtype=torch.float64,
              names=("vorticity", "u_z", "u_r"))
    work = _scratch(2 * nr, nz, vorticity.device)
    N.call("axi_advect_particles_f64", N.ptr(z_particles), N.ptr(r_particles),
           N.ptr(vort_particles), N.ptr(vorticity), N.ptr(Z_double), N.ptr(R_double), N.ptr(u_z),
           N.ptr(u_r), nr, nz, float(dx), float(dt), int(periodic), N.ptr(work),
           N.stream_of(vorticity))
    _check(work, 2 * nr, nz, vorticity)


def advect_vorticity_via_particles(z_particles, r_particles, vort_particles, vorticity, Z_double,
                                   R_double, grid_size_r, u_z, u_r, dx, dt):
    """kernels/advect_particle.py:5-35 (unbounded remeshing)."""
    _advect(z_particles, r_particles, vort_particles, vorticity, Z_double, R_double, grid_size_r,
            u_z, u_r, dx, dt, False)


def advect_vorticity_via_particles_periodic(z_particles, r_particles, vort_particles, vorticity,
                                            Z_double, R_double, grid_size_r, u_z, u_r, dx, dt):
    """kernels/advect_particle.py:38-68 (periodic remeshing)."""
    _advect(z_particles, r_particles, vort_particles, vorticity, Z_double, R_double, grid_size_r,
            u_z, u_r, dx, dt, True)
