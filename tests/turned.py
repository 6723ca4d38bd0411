"""A cavity whose elements start at a corner of their own (each quad's nodes turned by 0 to 3 places):
the same mesh, but neighbours meet along any pair of faces and in both directions, as on an
unstructured mesh."""

import os

import numpy as np

from ho2d import meshgen


def turned_cavity(outdir, n, knod, jitter=0.1, seed=5, steps=1):
    mesh = meshgen.cavity(n, jitter=jitter, seed=seed)
    turn = np.random.Generator(np.random.PCG64(seed + 1)).integers(0, 4, mesh.n_el)
    mesh.quads = np.stack([np.roll(q, k) for q, k in zip(mesh.quads, turn)])
    os.makedirs(outdir, exist_ok=True)
    meshgen.write_msh(mesh, os.path.join(outdir, "mesh.msh"))
    path = os.path.join(outdir, "input.dat")
    meshgen.write_input_dat(path, "mesh.msh", knod, 100.0, 1e-3, steps, 1)
    return path


def reversed_faces(c):
    """Interior faces of an oracle case that their two elements run through in opposite directions."""
    ijp = np.arange(4)[None, :]
    rev = (ijp + c.f_nijp - ijp // 2 - c.f_nijp // 2 + 1) % 2
    return (c.f_nbr >= 0) & (rev == 1)
