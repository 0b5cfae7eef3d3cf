"""Grid2D: drop-in for src/Grid.py:198-376, Cartesian or r-z.

Node arrays live on the GPU as torch tensors (torch is used only for device
memory).  ``rho`` is float32 charge density (C/m^3), ``phi`` FP64 potential,
``E`` float32 (2, m*n) field, ``b`` FP64 Poisson right-hand side.  Index
layout as the reference: idx = j*m + i with m nodes in x (src/Grid.py:140).

cylindrical=True is the axisymmetric r-z grid (src/Grid.py:5-93): x (m
nodes) is the axis z, y (n nodes, rows) the radius, row 0 on the axis.  The
deposit is divided by the node volumes of the linear weighting (so a uniform
load gives a uniform density), and E_r vanishes on the axis.  The reference
divides by ring volumes indexed along the wrong axis and does not zero E_r
there (src/Grid.py:66-93).
"""
from __future__ import annotations

import numpy as np
import torch

from . import _lib

DEVICE = "cuda"

# From so many particles per node, and so many in all, the deposit goes through
# the cells' corner sums and the gather through node pairs (particles.cu): below,
# clearing and summing the scratch costs what the particles save.  Pairs stop at
# PAIR_NODES nodes (8 MiB): past them sorted particles gather faster from the
# planes (16M sorted particles on 2049^2 nodes: 107 us against 118).
DENSE_PER_NODE, DENSE_PARTICLES, PAIR_NODES = 2, 400_000, 1 << 19


class Grid2D:
    """Grid2D(m, n, X, Y) -- m, n are NODE counts; dx = X/(m-1) (src/Grid.py:199-228)."""

    def __init__(self, m, n, X, Y, cylindrical=False):
        self.cylindrical = bool(cylindrical)
        self.m = int(m)
        self.n = int(n)
        self.X = float(X)
        self.Y = float(Y)
        self.dx = self.X / (self.m - 1)
        self.dy = self.Y / (self.n - 1)
        self.gridshape = (self.m, self.n)
        self.node_count = self.m * self.n
        self.cell_size = (self.dx, self.dy)
        self.cell_count = (self.m - 1) * (self.n - 1)
        self.domain = (self.X, self.Y)
        G = self.node_count
        self.rho = torch.zeros(G, dtype=torch.float32, device=DEVICE)
        self.b = torch.zeros(G, dtype=torch.float64, device=DEVICE)
        self.phi = torch.zeros(G, dtype=torch.float64, device=DEVICE)
        self.E = torch.zeros((2, G), dtype=torch.float32, device=DEVICE)
        self._cells = self._pairs = None  # scratch of the dense deposit and gather, made at first use

    def update_E(self):
        """E = -grad(phi) (src/Grid.py:232-243); r-z: E_r = 0 on the axis."""
        _lib.call("pic_update_E_rz" if self.cylindrical else "pic_update_E", _lib.ptr(self.phi), _lib.ptr(self.E[0]),
                  _lib.ptr(self.E[1]), self.m, self.n, self.dx, self.dy, _lib.stream_ptr())

    def update_density(self, particles):
        """CIC charge deposit of every species, rho in C/m^3 (src/Grid.py:246-294);
        r-z: divided by the node volumes (pic_rz_density)."""
        if self._dense(particles) and self._scratch("_cells"):
            self._cells.zero_()
            fn, target = "pic_deposit_cells", self._cells
        else:
            self.rho.zero_()
            fn, target = "pic_deposit", self.rho
        for s in particles.species:
            if s.n == 0:
                continue
            scale = s.charge * particles.species_np2c(s) / (self.dx * self.dy)
            _lib.call(fn, _lib.ptr(s.x), _lib.ptr(s.y), s.n, scale, _lib.ptr(target), self.m, self.n,
                      _lib.stream_ptr())
        if target is self._cells:
            _lib.call("pic_cells_density", _lib.ptr(self._cells), _lib.ptr(self.rho), self.m, self.n,
                      _lib.stream_ptr())
        if self.cylindrical:
            _lib.call("pic_rz_density", _lib.ptr(self.rho), self.m, self.n, self.dy, _lib.stream_ptr())

    def _dense(self, particles):
        n = sum(s.n for s in particles.species)
        return n >= max(DENSE_PARTICLES, DENSE_PER_NODE * self.node_count)

    def _scratch(self, name):
        """Whether the dense path's scratch is there: made at first use, if the device has room for it."""
        if getattr(self, name) is None:
            try:
                setattr(self, name, torch.empty((self.node_count, 4), dtype=torch.float32, device=DEVICE))
            except torch.OutOfMemoryError:
                return False
        return True

    def field_pairs(self, particles):
        """E as node pairs (pic_field_pairs) for the gather of `particles`, or None where the planes serve better."""
        if self.node_count > PAIR_NODES or not self._dense(particles) or not self._scratch("_pairs"):
            return None
        _lib.call("pic_field_pairs", _lib.ptr(self.E[0]), _lib.ptr(self.E[1]), _lib.ptr(self._pairs), self.m, self.n,
                  _lib.stream_ptr())
        return self._pairs

    def update_J(self, particles):
        pass

    def minmax_phi(self):
        return torch.min(self.phi), torch.max(self.phi)

    def minmax_rho(self):
        return torch.min(self.rho), torch.max(self.rho)

    def save_to_txt(self, filename, fields=None, header=None):
        """Columns x, y, fields... in '%.2e' (the format of src/Grid.py:306-375)."""
        if fields is None:
            fields = {"rho": self.rho, "phi": self.phi, "E_x": self.E[0], "E_y": self.E[1]}
        j, i = np.divmod(np.arange(self.node_count), self.m)
        cols = [i * self.dx, j * self.dy]
        names = []
        for name, f in fields.items():
            names.append(name)
            cols.append(f.detach().cpu().numpy() if isinstance(f, torch.Tensor) else np.asarray(f))
        if header is None:
            header = "x y " + " ".join(names)
        np.savetxt(filename, np.column_stack(cols), header=header, comments="# ", fmt="%.2e")
