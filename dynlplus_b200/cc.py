"""Connected components on the device (dynlp/cc.py:8-23).

`connected_components(n, rows, cols)` returns (int32 labels in [0, n_comp), n_comp) with the
reference's canonical numbering: components ranked by their smallest vertex id (the reference's
`unique(..., return_inverse=True)` relabel, cc.py:22). The kernel is a lock-free union-find
(hook larger root under smaller, path halving) rather than the reference's host-synchronised
hook/jump rounds; the labels are identical bit for bit.
"""
from __future__ import annotations

import torch

from . import _lib
from .backend import code, ptr, stream, workspace


def _roots(n, rows, cols, err) -> torch.Tensor:
    rows = rows.to(torch.int32).contiguous()
    cols = cols.to(torch.int32).contiguous()
    parent = torch.empty(max(n, 1), dtype=torch.int32, device=rows.device)
    ws = workspace("cc_edges").get(_lib.lib().dlp_cc_edges_workspace_bytes())
    _lib.call("dlp_cc_edges_ws", int(n), ptr(rows), ptr(cols), int(rows.numel()), ptr(parent), ptr(err), ptr(ws),
              ws.numel(), stream())
    return parent[:n]


def _raise_on(err):
    if err < 0:
        raise _lib.DLPError("dlp_cc_edges_ws", -err)
    if err:
        raise ValueError("connected_components: edge endpoint outside [0, n)")


def min_vertex_roots(n, rows, cols) -> torch.Tensor:
    """parent[v] = smallest vertex id in v's component (int32, device)."""
    err = torch.zeros(1, dtype=torch.int32, device=rows.device)
    parent = _roots(n, rows, cols, err)
    _raise_on(int(err.item()))
    return parent


def relabel(parent: torch.Tensor, sync: bool = True, count=None):
    """Rank of each root among the roots (unique + inverse); returns (labels, n_comp). count: where the
    component count goes (device int32[1])."""
    n = int(parent.numel())
    label = torch.empty(max(n, 1), dtype=torch.int32, device=parent.device)
    nc = torch.empty(1, dtype=torch.int32, device=parent.device) if count is None else count
    ws = workspace("compact").get(_lib.lib().dlp_compact_workspace_bytes(n))
    _lib.call("dlp_cc_relabel", n, ptr(parent), ptr(label), ptr(nc), ptr(ws), ws.numel(), stream())
    return (label[:n], int(nc.item())) if sync else (label[:n], nc)


def connected_components(n, rows, cols):
    """(labels in [0, n_comp), n_comp) for an undirected edge list (dynlp/cc.py:8-23). One host read."""
    if n == 0:
        dev = rows.device if torch.is_tensor(rows) else None
        return torch.zeros(0, dtype=torch.int32, device=dev), 0
    ec = torch.zeros(2, dtype=torch.int32, device=rows.device)  # [error, count]
    label, _ = relabel(_roots(n, rows, cols, ec[:1]), sync=False, count=ec[1:])
    err, nc = ec.tolist()
    _raise_on(err)
    return label, nc


def graph_components(G, vmask=None, sink=None, w=None):
    """Min-vertex-id roots over the stored entries of a row-range graph with a sink vertex n.

    Entry (u, v) joins u and v when vmask[u] and vmask[v] (and w != 0 when w is given); it joins
    u and the sink when vmask[u] and sink[v]. Returns parent of length n + 1 (device int32).
    This is the grounding check of dynlp/stream.py:150-159 and :275-280 in one launch.
    """
    n = G.shape[0]
    dev = G.indices.device
    parent = torch.empty(n + 1, dtype=torch.int32, device=dev)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    ws = workspace("cc_graph").get(_lib.lib().dlp_cc_graph_workspace_bytes())
    _lib.call("dlp_cc_graph", n, ptr(G.rbeg), ptr(G.rend), ptr(G.indices), ptr(w),
              code(w) if w is not None else 0, ptr(vmask), ptr(sink), ptr(parent), ptr(err), ptr(ws), ws.numel(),
              stream())
    return parent, err


def ground_reach(G, vmask, sink, umask, in_t, w=None):
    """Grounded set of the graph form of graph_components, updated in place: umask[u] = 1 iff
    vmask[u] and u's component reaches the sink (the vertices whose root is the sink's root there);
    in_t[u] = 1 where membership changed. Bottom-up reachability sweeps; the union-find finishes
    the job when they do not settle. Returns (number of changes, sweeps run; negative = fallback)."""
    import ctypes as ct
    n = G.shape[0]
    dev = G.indices.device
    ce = torch.zeros(2, dtype=torch.int32, device=dev)  # [changes, error]: read back together
    cnt, err = ce[0:1], ce[1:2]
    sweeps = ct.c_int32(0)
    ws = workspace("ground_reach").get(_lib.lib().dlp_ground_reach_workspace_bytes(n))
    rbeg, rend = (G.rbeg, G.rend) if hasattr(G, "rbeg") else (G.indptr[:-1], G.indptr[1:])
    _lib.call("dlp_ground_reach", n, ptr(rbeg), ptr(rend), ptr(G.indices), ptr(w), code(w) if w is not None else 0,
              ptr(vmask), ptr(sink), ptr(umask), ptr(in_t), ptr(cnt), ptr(err), ct.addressof(sweeps), ptr(ws),
              ws.numel(), stream())
    changes, bad = ce.tolist()
    if bad:
        raise ValueError("ground_reach: entry column outside [0, n)")
    return changes, int(sweeps.value)



# ---------------------------------------------------------------------------------------------
# adaptive components of new vertices (dynlp/cc.py:26-83)
# ---------------------------------------------------------------------------------------------
def _ids32(ids):
    """int32 ids; one past int32 becomes its lowest or highest value, out of range for the kernel too."""
    if ids.dtype == torch.int64:
        ids = ids.clamp(-2**31, 2**31 - 1)
    return ids.to(torch.int32).contiguous()


def fh_components(m, rows, cols, d, k, ground=None):
    """Felzenszwalb-Huttenlocher merging in Boruvka rounds (dynlp/cc.py:37-73): each round every
    component takes its lightest outgoing edge (ties to the smallest other side) and merges across it
    when d(e) <= min over both sides of Int(C) + k/|C| (Int = largest internal dissimilarity, fp32 as
    the reference keeps it); with `ground`, components holding none then join their lightest neighbour
    until every one has some. One launch (dlp_fh_components) and the rank labels."""
    dev = rows.device
    if m == 0 or not rows.numel():
        return torch.arange(m, dtype=torch.int32, device=dev), m
    if cols.shape != rows.shape or d.shape != rows.shape or rows.dim() != 1:
        raise IndexError(f"{tuple(rows.shape)}, {tuple(cols.shape)} and {tuple(d.shape)} edge ends and weights")
    if ground is not None and ground.shape != (m,):
        raise IndexError(f"ground of shape {tuple(ground.shape)} for {m} vertices")
    rows, cols = _ids32(rows), _ids32(cols)
    d = d.to(torch.float32).contiguous()
    g = ground.to(torch.float32).contiguous() if ground is not None else None
    root = torch.empty(m, dtype=torch.int32, device=dev)
    ec = torch.zeros(2, dtype=torch.int32, device=dev)  # [error, component count]
    ws = workspace("fh").get(_lib.lib().dlp_fh_components_workspace_bytes(m))
    _lib.call("dlp_fh_components", int(m), int(rows.numel()), ptr(rows), ptr(cols), ptr(d), float(k), ptr(g), ptr(root),
              ptr(ec), ptr(ws), ws.numel(), stream())
    lab, _ = relabel(root, sync=False, count=ec[1:])
    err, nc = ec.tolist()
    if err == _lib.DLP_ERR_INVALID:
        raise IndexError(f"fh_components: edge end outside [0, {m})")
    if err:
        raise _lib.DLPError("dlp_fh_components", err)
    return lab, nc


def adaptive_components(m, rows, cols, w, s_r, s_c, wmax, ground=None):
    """Component-adaptive merging of the new vertices (dynlp/cc.py:76-83): dissimilarity
    1 - w/wmax scaled by the endpoints' own mean dissimilarities, k = its mean."""
    if m == 0:
        return torch.zeros(0, dtype=torch.int32, device=rows.device), 0
    d = (1 - w / wmax) / torch.sqrt(s_r * s_c)
    k = float(d.double().mean().item()) if d.numel() else 0.0
    return fh_components(m, rows, cols, d, k, ground)
