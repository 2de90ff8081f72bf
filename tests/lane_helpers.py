"""Shared by the lane kernels' GPU tests: which kernel a handle has, and mesh files of
tensor-product grids with any node positions."""
import numpy as np

import hpgem_b200


def kernel_class(solver):
    """The kernel class a batch takes the handle in: "lane tables" (simplices and the wave)
    and "sum-factorised lanes" are the lane kernels, the others the general ones."""
    batch = hpgem_b200.Batch(1)
    slot = batch.add(solver, 1e-6, 0)
    kind = batch.class_info()[0]["kind"]
    batch.remove(slot)
    batch.close()
    return kind


def write_mesh_file(path, axes, triangles=False, jiggle=0.0):
    """A periodic "mesh 2" file: nodes at the products of `axes` (each from the lower to the
    upper corner, both included), each then moved by up to `jiggle` cells of its own;
    quadrilaterals, hexahedra or two triangles per cell."""
    rng = np.random.default_rng(7)
    dim, cells = len(axes), [len(a) - 1 for a in axes]
    number = {}
    lines = []
    for idx in np.ndindex(*cells[::-1]):
        idx = idx[::-1]
        number[idx] = len(number)
        wraps = [c for c in range(dim) if idx[c] == 0]
        off = [jiggle * rng.uniform(-1.0, 1.0) * (axes[c][-1] - axes[c][0]) / cells[c] for c in range(dim)]
        copies = []
        for sub in range(1 << len(wraps)):
            far = [c for b, c in enumerate(wraps) if sub >> b & 1]
            copies.append([axes[c][cells[c] if c in far else idx[c]] + off[c] for c in range(dim)])
        lines += ["1 0", "%d %s" % (len(copies), " ".join(float(v).hex() for x in copies for v in x))]
    corners = [[0, 1, 2], [1, 3, 2]] if triangles else [list(range(1 << dim))]
    elements = []
    for idx in np.ndindex(*cells[::-1]):
        idx = idx[::-1]
        for element in corners:
            words = [str(len(element))]
            for v in element:
                at = [idx[c] + (v >> c & 1) for c in range(dim)]
                node = tuple(at[c] % cells[c] for c in range(dim))
                wraps = [c for c in range(dim) if node[c] == 0]
                copy = sum(1 << b for b, c in enumerate(wraps) if at[c] == cells[c])
                words += [str(number[node]), str(copy)]
            elements += [" ".join(words + ["0"]), "0"]
    head = ["mesh 2", "%d %d %d 0" % (len(number), len(elements) // 2, dim), "1 %d" % (len(elements) // 2), "zones", "1", "Main", "nodes"]
    path.write_text("\n".join(head + lines + ["elements"] + elements) + "\n")
    return path
