"""Kernels at the sizes where a tile, a remainder or a dispatch rule can go wrong, against the same sums in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
U = 2.0 ** -24   # unit roundoff of float32


def _linear64(W, x, inds):
    r = x.double().reshape(x.shape[0], x.shape[1], -1)
    return torch.einsum("oi,ris->ros", W.double(), r).reshape(x.shape[0], W.shape[0], *x.shape[2:])


# rows that leave ragged tiles on both sides of the small-tile rule (a tile holds 16 to 512 rows, 148 blocks), widths around
# the 32 / 64 / 128 outputs of a tile and the 8 / 16 channels of a step
@pytest.mark.parametrize("inds", [0, 1, 2])
@pytest.mark.parametrize("rows,dim_in,dim_out", [(1, 1, 1), (15, 7, 33), (513, 17, 32), (3001, 24, 65), (2500, 9, 129), (20003, 8, 31),
                                                 (9500, 40, 64)])
def test_tensor_linear_tiles(inds, rows, dim_in, dim_out):
    from ld_b200 import ops
    g = torch.Generator().manual_seed(rows + inds)
    W = torch.randn(dim_out, dim_in, generator=g)
    x = torch.randn(rows, dim_in, *[3] * inds, generator=g)
    dy = torch.randn(rows, dim_out, *[3] * inds, generator=g)
    y = ops.tensor_linear_fwd(inds, W.cuda(), x.cuda()).cpu().double()
    # a sum of n products in any order, with FMAs: |error| <= n u sum |w||x|
    bound = dim_in * U * _linear64(W.abs(), x.abs(), inds)
    assert bool(((y - _linear64(W, x, inds)).abs() <= bound).all())
    yt = ops.tensor_linear_fwd(inds, W.cuda().t(), dy.cuda()).cpu().double()   # strided weights
    assert bool(((yt - _linear64(W.t(), dy, inds)).abs() <= dim_out * U * _linear64(W.t().abs(), dy.abs(), inds)).all())
    dW = ops.tensor_linear_dw(inds, dy.cuda(), x.cuda(), dim_out, dim_in).cpu().double()
    flat = lambda t: t.double().reshape(rows, t.shape[1], -1)  # noqa: E731
    want = torch.einsum("ros,ris->oi", flat(dy), flat(x))
    size = torch.einsum("ros,ris->oi", flat(dy).abs(), flat(x).abs())
    assert bool(((dW - want).abs() <= rows * 3 ** inds * U * size).all())


@pytest.mark.parametrize("rows,chan", [(1, 1), (5, 7), (3, 32), (41, 33), (9000, 136)])   # warps with missing lanes, grid strides
def test_bee_products_tails(rows, chan):
    from ld_b200 import ops
    from oracle import reference_math as R
    g = torch.Generator().manual_seed(rows)
    t = [torch.randn(rows, chan, *[3] * (k % 3), generator=g) for k in range(6)]
    got = ops.bee_fwd(*[a.cuda() for a in t])
    want = R.bee(*[a.double() for a in t])
    size = R.bee(*[a.double().abs() for a in t])
    for k, (a, b, m) in enumerate(zip(got, want, size)):
        if k in (11, 12):   # cross products: both terms count with their size
            m = b.abs() + 2 * (t[1] if k == 11 else t[2]).double().abs().amax(-1, keepdim=True) * t[4].double().abs().amax(-1).reshape(
                rows, chan, *[1] * (k - 10))
        assert bool(((a.cpu().double() - b).abs() <= 10 * U * m).all()), k


def _message64(row_ptr, dst, rij, weights, actv, x_v, radial, n_rbf, rmax):
    from oracle import reference_math as R
    (W1, b1), (W2, b2), (W3, b3) = [(W.double(), b.double()) for W, b in weights]
    n = x_v.shape[1]
    r = rij.double()
    h = (R.radial_encode_painn if radial == 0 else R.radial_encode_gaussian)(r, n_rbf, rmax)
    silu = torch.nn.functional.silu
    P = (silu(silu(h @ W1.t() + b1) @ W2.t() + b2) @ W3.t() + b3) * actv.double()[dst.long()]
    u = (r / torch.sqrt(0.1 + (r ** 2).sum(-1, keepdim=True)))[:, None]
    xe = x_v.double()[dst.long()]
    m = xe * P[:, :n, None] + torch.linalg.cross(xe, u.expand_as(xe)) * P[:, n:2 * n, None] + u * P[:, 2 * n:3 * n, None]
    src = torch.repeat_interleave(torch.arange(len(row_ptr) - 1), (row_ptr[1:] - row_ptr[:-1]).long())
    zeros = torch.zeros(x_v.shape, dtype=torch.float64)
    return zeros[..., 0].index_add(0, src, P[:, 3 * n:]), zeros.index_add(0, src, m)


# tiles hold 256, 128 or 64 edges (n = 32, 64, 128), slabs K = 32: nodes without edges, nodes that span tiles, a last tile
# with one edge, input widths around the slab; weights far from 1 move the operands' scales
@pytest.mark.parametrize("n,n_rbf,radial,degrees,wscale", [
    (32, 1, 1, "one", 1.0), (32, 20, 1, "mixed", 1.0), (32, 128, 0, "long", 1.0), (64, 16, 1, "long", 30.0), (64, 64, 0, "mixed", 1.0),
    (128, 8, 1, "mixed", 1.0), (128, 33, 0, "long", 1e-3), (128, 16, 1, "none", 1.0)])
def test_split_message_is_as_exact_as_the_fma_kernel(n, n_rbf, radial, degrees, wscale):
    """the two kernels against 64 bits: the split form may not be further off than the FP32 FMAs are (plus one rounding)"""
    import ctypes
    from ld_b200 import ops
    from ld_b200._lib import lib, check, ptr, stream_ptr
    g = torch.Generator().manual_seed(n + n_rbf)
    deg = {"one": torch.tensor([0, 0, 1, 0]), "none": torch.zeros(5, dtype=torch.int64),
           "mixed": torch.randint(0, 40, (61,), generator=g), "long": torch.tensor([3, 0, 700, 1, 0, 0, 64, 257, 129, 1])}[degrees]
    Nt, E = len(deg), int(deg.sum())
    row_ptr = torch.cat([torch.zeros(1, dtype=torch.int64), deg.cumsum(0)]).int()
    dst = torch.randint(0, Nt, (E,), generator=g).int()
    rmax = 4.0
    rij = torch.randn(E, 3, generator=g) * 1.3
    lin = [torch.nn.Linear(k, 4 * n) for k in (n_rbf, 4 * n, 4 * n)]
    with torch.no_grad():
        for l in lin:
            l.weight.copy_((torch.rand(l.weight.shape, generator=g) * 2 - 1) * l.weight.shape[1] ** -0.5 * wscale)
            l.bias.copy_((torch.rand(l.bias.shape, generator=g) * 2 - 1) * l.weight.shape[1] ** -0.5)
    actv, x_v = torch.randn(Nt, 4 * n, generator=g), torch.randn(Nt, n, 3, generator=g)
    want = _message64(row_ptr, dst, rij, [(l.weight.detach(), l.bias.detach()) for l in lin], actv, x_v, radial, n_rbf, rmax)
    mlp = ops.PackedMLP([l.cuda() for l in lin])
    args = [t.cuda() for t in (row_ptr, dst, rij)]
    actv, x_v = actv.cuda(), x_v.cuda()
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    split = ops.painn_message_f32(*args, mlp, actv, x_v, rmax, radial_kind=radial, edge_counter=count)
    assert mlp._split and int(count) == E and int(ops.tc_status(actv.device)) == 0
    fma = torch.empty(Nt, n, device="cuda"), torch.empty(Nt, n, 3, device="cuda")
    check(lib().ld_painn_message_f32(*[ptr(a) for a in args], Nt, n, n_rbf, radial, ctypes.c_float(rmax), ctypes.c_float(0.1), ptr(mlp.Wt[0]),
                                     ptr(mlp.b[0]), ptr(mlp.Wt[1]), ptr(mlp.b[1]), ptr(mlp.Wt[2]), ptr(mlp.b[2]), ptr(actv), ptr(x_v), None,
                                     None, ptr(fma[0]), ptr(fma[1]), None, stream_ptr()))
    for w, a, b in zip(want, split, fma):
        off = lambda t: float((t.cpu().double() - w).norm())  # noqa: E731
        assert off(a) <= 1.2 * off(b) + U * float(w.norm()), (off(a) / float(w.norm()), off(b) / float(w.norm()))

# tiles of 128 edges, at n = 128 taken in two passes of 64; slabs K = 64: input widths around them, nodes without edges and
# nodes that span tiles, one edge in the last tile
@pytest.mark.parametrize("n,n_rbf,radial,degrees", [(32, 1, 1, "one"), (32, 128, 0, "long"), (64, 65, 0, "mixed"), (64, 16, 1, "long"),
                                                    (128, 8, 1, "mixed"), (128, 80, 0, "long"), (128, 16, 1, "none")])
def test_bf16_slab_message_against_the_edge_major_kernel(n, n_rbf, radial, degrees):
    """both BF16 kernels against 64 bits: the slab kernel (which reads the features in FP32) may not be further off, plus one
    rounding to BF16 of what is summed"""
    import ctypes
    from ld_b200 import ops
    from ld_b200._lib import lib, check, ptr, stream_ptr
    g = torch.Generator().manual_seed(n + n_rbf)
    deg = {"one": torch.tensor([0, 0, 1, 0]), "none": torch.zeros(5, dtype=torch.int64),
           "mixed": torch.randint(0, 40, (61,), generator=g), "long": torch.tensor([3, 0, 700, 1, 0, 0, 64, 257, 129, 1])}[degrees]
    Nt, E = len(deg), int(deg.sum())
    row_ptr = torch.cat([torch.zeros(1, dtype=torch.int64), deg.cumsum(0)]).int()
    dst = torch.randint(0, Nt, (E,), generator=g).int()
    rij = torch.randn(E, 3, generator=g) * 1.3
    torch.manual_seed(n)
    lin = [torch.nn.Linear(k, 4 * n) for k in (n_rbf, 4 * n, 4 * n)]
    actv, x_v = torch.randn(Nt, 4 * n, generator=g), torch.randn(Nt, n, 3, generator=g)
    want = _message64(row_ptr, dst, rij, [(l.weight.detach(), l.bias.detach()) for l in lin], actv, x_v, radial, n_rbf, 4.0)
    mlp = ops.PackedMLP([l.cuda() for l in lin])
    args = [t.cuda() for t in (row_ptr, dst, rij)]
    actv, x_v = actv.cuda(), x_v.cuda()
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    res = torch.randn(Nt, n, generator=g).cuda(), torch.randn(Nt, n, 3, generator=g).cuda()
    slabs = ops.painn_message_bf16_tc(*args, mlp, actv, x_v, 4.0, radial_kind=radial, edge_counter=count)
    added = ops.painn_message_bf16_tc(*args, mlp, actv, x_v, 4.0, radial_kind=radial, res_a=res[0], res_v=res[1])
    assert mlp._slabs and int(count) == E and int(ops.tc_status(actv.device)) == 0
    w = ops._packed_bf16(mlp)
    old = torch.empty(Nt, n, device="cuda"), torch.empty(Nt, n, 3, device="cuda")
    check(lib().ld_painn_message_bf16_tc(*[ptr(a) for a in args], Nt, n, n_rbf, radial, ctypes.c_float(4.0), ctypes.c_float(0.1), ptr(w[0]),
                                         ptr(mlp.b[0]), ptr(w[1]), ptr(mlp.b[1]), ptr(w[2]), ptr(mlp.b[2]), ptr(actv), ptr(x_v), None, None,
                                         None, ptr(old[0]), ptr(old[1]), None, ptr(ops.tc_status(actv.device)), stream_ptr()))
    for w64, a, b, r, ar in zip(want, slabs, old, res, added):
        off = lambda t: float((t.cpu().double() - w64).norm())  # noqa: E731
        assert off(a) <= 1.2 * off(b) + 2.0 ** -9 * float(w64.norm()), (off(a) / float(w64.norm()), off(b) / float(w64.norm()))
        assert torch.equal(ar, a + r)


# tiles of 64 edges, groups of 16: nodes without edges, nodes that span tiles, one edge in the last tile; both widths of
# either kind of channel; sizes of the features that move the scales of the operands, one edge far above the others
@pytest.mark.parametrize("chan,dim_a,degrees,size", [(128, 128, "mixed", 1.0), (128, 64, "long", 1.0), (64, 128, "mixed", 1e6),
                                                     (64, 64, "long", 1e-5), (128, 128, "one", 1.0), (64, 64, "none", 1.0), (128, 128, "long", "spread")])
def test_split_scalar_channel_is_as_exact_as_the_fma_kernel(chan, dim_a, degrees, size):
    from ld_b200 import bee
    from ld_b200.graph_layers import Graph
    from ld_b200._lib import lib, check, ptr, stream_ptr
    from ld_b200 import ops
    g = torch.Generator().manual_seed(chan + dim_a)
    deg = {"one": torch.tensor([0, 0, 1, 0]), "none": torch.zeros(5, dtype=torch.int64),
           "mixed": torch.randint(0, 40, (61,), generator=g), "long": torch.tensor([3, 0, 300, 1, 0, 0, 64, 17, 129, 16])}[degrees]
    Nt, E = len(deg), int(deg.sum())
    src = torch.repeat_interleave(torch.arange(Nt), deg)
    dst = torch.randint(0, Nt, (E,), generator=g)
    rij = torch.randn(E, 3, generator=g) * 1.5
    torch.manual_seed(3)
    m = bee.Messages(5.0, dim_a, 32, 32, chan).cuda()
    rows = torch.randn(Nt, 13, chan, generator=g)
    if size == "spread":
        rows *= 10.0 ** torch.randint(-8, 8, (Nt, 1, 1), generator=g)
    else:
        rows *= size
    graph = Graph(src.cuda(), dst.cuda(), None, 1, Nt)
    with torch.no_grad():
        w = m._pack()
    r13, rc = rows.cuda(), rij.cuda()
    l = [r13[:, 0].contiguous(), r13[:, 1:4].transpose(1, 2).contiguous(), r13[:, 4:].transpose(1, 2).contiguous()]
    again = torch.empty_like(r13)
    check(lib().ld_bee_rows13_f32(ptr(l[0]), ptr(l[1]), ptr(l[2]), Nt, chan, ptr(again), stream_ptr()))
    assert torch.equal(again, r13)
    split, fma = torch.full((Nt, dim_a), 7.0, device="cuda"), torch.full((Nt, dim_a), 7.0, device="cuda")
    geo = (ptr(graph.row_ptr), ptr(graph.dst32), ptr(rc), Nt, chan, dim_a, 5.0)
    enc = (ptr(w["enc_w"]), ptr(w["enc_b"]), ptr(w["jac"]))
    check(lib().ld_bee_messages_scalar_f32_split(*geo, ptr(r13), *enc, ptr(w["split"]), ptr(w["split_scales"]), ptr(w["b1"]), ptr(w["b2"]),
                                                 ptr(w["b3"]), 0.1, ptr(split), ptr(ops.tc_status(r13.device)), stream_ptr()))
    check(lib().ld_bee_messages_scalar_f32(*geo, *[ptr(t) for t in l], *enc, ptr(w["Yt"]), ptr(w["W1t"]), ptr(w["b1"]), ptr(w["W2t"]),
                                           ptr(w["b2"]), ptr(w["W3t"]), ptr(w["b3"]), ptr(w["Wdt"]), 0.1, ptr(fma), stream_ptr()))
    assert int(ops.tc_status(r13.device)) == 0
    # the same layer in 64 bits
    p = {k: v.detach().cpu().double() for k, v in m.state_dict().items()}
    r = rij.double()
    phi = bee.radial_encode_8(r, 5.0) @ p["lin_enc.weight"].t() + p["lin_enc.bias"]
    u = r * 1.4
    u = u / torch.sqrt(1 + (u ** 2).sum(-1, keepdim=True))
    f = rows.double()[dst]
    y = [f[:, 0] * phi, torch.einsum("ekc,ek->ec", f[:, 1:4], u) * phi,
         torch.einsum("exyc,ex,ey->ec", f[:, 4:].reshape(E, 3, 3, chan), u, u) * phi]
    psi = sum(t @ p[f"Y_{k}.W"].t() for t, k in zip(y, ("000", "110", "220")))
    h = psi
    for k in (0, 2, 4):
        h = h @ p[f"mlp_a.layers.{k}.weight"].t() + p[f"mlp_a.layers.{k}.bias"]
        h = torch.nn.functional.leaky_relu(h, 0.1) if k < 4 else h
    want = torch.zeros(Nt, dim_a, dtype=torch.float64).index_add(0, src, 0.1 * (psi + psi @ p["mlp_a.lin_direct.weight"].t() + h))
    # per node (the sizes differ by orders of magnitude): not further off than the FMAs, plus a rounding of the largest edge
    edge = (0.1 * (psi.abs() + h.abs())).amax(-1)
    biggest = torch.zeros(Nt, dtype=torch.float64).index_reduce(0, src, edge, "amax")
    a, b = ((t.cpu().double() - want).norm(dim=-1) for t in (split, fma))
    assert bool((a <= 1.5 * b + 4 * U * biggest * dim_a ** 0.5 + 1e-30).all()), (a / (b + 1e-300)).max()


def test_split_kernels_give_a_node_the_same_bits_in_any_partition():
    """the outputs of a system do not depend on which systems are computed beside it"""
    from ld_b200 import bee, painn
    from ld_b200.graph_layers import Graph
    g = torch.Generator().manual_seed(5)
    B, N = 5, 37
    pos = torch.cumsum(torch.randn(B, N, 3, generator=g) / 3 ** 0.5, dim=1).cuda()
    feats = [torch.randn(B, N, *s, generator=g).cuda() for s in ((64,), (64, 3), (32, 3, 3))]
    torch.manual_seed(2)
    layer, message = bee.Messages(4.0, 64, 64, 32, 64).cuda(), painn.Message(4.0, 64).cuda()

    def run(lo, hi):
        graph = Graph.radius_graph(4.0, None, pos[lo:hi])
        x = [f[lo:hi] for f in feats]
        return (*layer(graph, graph.rij, *x), *message(graph, x[0], x[1], graph.rij, residual=True))

    with torch.no_grad():
        whole, parts = run(0, B), [run(0, 2), run(2, 3), run(3, B)]
    for k, w in enumerate(whole):
        assert torch.equal(w, torch.cat([p[k] for p in parts])), k


# one block per system up to 8192 nodes and cells (256 threads to 512 nodes), all particles together beyond; the degrees in one
# block up to 16384 nodes; boxes with two to many cells per axis, coordinates on the boundary and in other images
@pytest.mark.parametrize("batch,nodes,box,cutoff", [
    (3, 512, None, 3.0), (2, 513, (9.0, 7.0, 11.0), 2.9), (2, 8192, (20.0, 21.0, 22.0), 1.5), (1, 8193, (18.0, 20.0, 19.0), 1.4),
    (40, 410, (8.0, 8.0, 8.0), 1.1), (5, 37, (4.0, 4.1, 9.0), 1.9), (2, 300, (30.0, 60.0, 30.0), 1.0), (1, 1, None, 1.0)])
def test_radius_graph_build_paths(batch, nodes, box, cutoff):
    from ld_b200 import graph as G
    g = torch.Generator().manual_seed(nodes)
    if box is None:
        pos = torch.cumsum(torch.randn(batch, nodes, 3, generator=g) / 3 ** 0.5, dim=1)
    else:
        L = torch.tensor(box)
        pos = torch.rand(batch, nodes, 3, generator=g) * L
        pos[:, :: 7] += L * torch.randint(-3, 4, pos[:, :: 7].shape, generator=g)
        pos[:, 1 :: 11, 0] = L[0]
        pos[:, 2 :: 11, 1] = 0.0
        pos[:, 3 :: 13, 2] = torch.nextafter(L[2], torch.zeros(()))
    b = G.RadiusGraphBuilder(batch, nodes, cutoff, box)
    got = b.build(pos.cuda(), want_shift=True)
    assert int(b.status) == 0
    from oracle import reference_math as R
    oracle = R.radius_graph(pos, cutoff, box)
    src, dst = oracle["src"], oracle["dst"]
    E = got["E"]
    key = lambda s, d: torch.sort(s.cpu().long() * (batch * nodes) + d.cpu().long()).values  # noqa: E731
    assert torch.equal(key(got["src"], got["dst"]), key(src, dst))
    deg = torch.bincount(got["src"].cpu().long(), minlength=batch * nodes)
    assert torch.equal(got["row_ptr"].cpu().long(), torch.cat([torch.zeros(1, dtype=torch.long), deg.cumsum(0)]))
    assert torch.equal(got["edge_counts"].cpu().long(), deg.reshape(batch, nodes).sum(1).cumsum(0))
    s, d = got["src"].cpu().long(), got["dst"].cpu().long()
    # displacements and shifts of the same pairs (the two lists order a node's neighbours differently)
    mine, ref = torch.argsort(s * (batch * nodes) + d), torch.argsort(src.long() * (batch * nodes) + dst.long())
    assert torch.equal(got["rij"].cpu()[mine], oracle["rij"][ref])
    assert torch.equal(G.unpack_shift(got["shift"]).cpu()[mine], oracle["shift"][ref].int())
    assert bool((s[1:] >= s[:-1]).all()) and E == len(src)


# 4, 8 or 16 rows per block with the line at 592 and 1184 rows; widths that leave threads over (192, 40) and the widest
@pytest.mark.parametrize("rows", [1, 5, 593, 1185, 2371])
@pytest.mark.parametrize("k0,n1,n2,n3,direct", [(64, 256, 256, 256, False), (128, 192, 192, 192, False), (7, 40, 8, 24, True), (512, 512, 512, 512, True)])
def test_mlp_rows_tiles(rows, k0, n1, n2, n3, direct):
    from ld_b200 import ops
    torch.manual_seed(rows + k0)
    lin = [torch.nn.Linear(a, b) for a, b in ((k0, n1), (n1, n2), (n2, n3))]
    d = torch.nn.Linear(k0, n3, bias=False) if direct else None
    x = torch.randn(rows, k0)
    y = ops.mlp3_rows(x.cuda(), ops.PackedMLP([l.cuda() for l in lin], None if d is None else d.cuda())).cpu().double()
    W = [(l.weight.detach().cpu().double(), l.bias.detach().cpu().double()) for l in lin]
    silu = torch.nn.functional.silu
    # first-order propagation of |error| <= (terms + 4) u (sum of sizes) through each layer (SiLU's slope is at most 1.1)
    h, e = x.double(), torch.zeros(rows, k0, dtype=torch.float64)
    for i, (w, b) in enumerate(W):
        size = h.abs() @ w.abs().t() + b.abs()
        e = e @ w.abs().t() + (w.shape[1] + 4) * U * size
        h = h @ w.t() + b
        if i < 2:
            h, e = silu(h), 1.1 * e + 4 * U * h.abs()
    if d is not None:
        wd = d.weight.detach().cpu().double()
        h, e = h + x.double() @ wd.t(), e + (k0 + w.shape[1] + 4) * U * (x.double().abs() @ wd.abs().t() + size)
    assert bool(((y - h).abs() <= e).all())


@pytest.mark.parametrize("n,batch,nodes", [(32, 1, 3), (64, 8, 64), (24, 2, 35)])
def test_painn_update_in_its_residual_form(n, batch, nodes):
    """the fused form against the module's own formula in 64 bits"""
    from ld_b200 import painn
    torch.manual_seed(n)
    m = painn.Update(n).cuda()
    x_a, x_v = torch.randn(batch, nodes, n).cuda(), torch.randn(batch, nodes, n, 3).cuda()
    p = {k: v.detach().double() for k, v in m.state_dict().items()}
    mix = lambda k: torch.einsum("oi,bnix->bnox", p[k], x_v.double())  # noqa: E731
    left, right = mix("lin_l.W"), mix("lin_r.W")
    y = torch.cat([x_a.double(), right.norm(dim=-1)], dim=-1)
    for k in (0, 2, 4):
        y = y @ p[f"mlp.layers.{k}.weight"].t() + p[f"mlp.layers.{k}.bias"]
        y = torch.nn.functional.silu(y) if k < 4 else y
    d_v = mix("lin_v.W") * y[..., :n, None]
    h = ((left * right).sum(-1) * y[..., n:2 * n]).reshape(batch, nodes, 4, n // 4)
    h = h - h.mean([1, 3], keepdim=True)
    h = (h / torch.sqrt(1 + (h ** 2).mean([1, 3], keepdim=True))).reshape(batch, nodes, n)
    want = x_a.double() + p["gn.beta"] + p["gn.gamma"] * h + y[..., 2 * n:], x_v.double() + d_v / torch.sqrt(1 + (d_v ** 2).sum(-1, keepdim=True))
    with torch.no_grad():
        got = m.residual(x_a, x_v)
        parts = m(x_a, x_v)
    for g, w, d, x in zip(got, want, parts, (x_a, x_v)):
        off = float((g.double() - w).norm() / w.norm())
        assert off <= 1.5 * float(((x + d).double() - w).norm() / w.norm()) + 2 * U, off   # not further off than the separate operations


def test_painn_update_reads_its_mixing_weights_in_every_call():
    """writes that autograd's version counter does not see (.data, another tensor at the same place) take effect at once"""
    from ld_b200 import painn
    torch.manual_seed(4)
    m = painn.Update(32).cuda()
    x_a, x_v = torch.randn(2, 17, 32).cuda(), torch.randn(2, 17, 32, 3).cuda()
    with torch.no_grad():
        m.residual(x_a, x_v)
        for name in ("lin_l", "lin_r", "lin_v"):
            getattr(m, name).W.data.mul_(-1.7)
            fresh = painn.Update(32).cuda()
            fresh.load_state_dict(m.state_dict())
            for a, b in zip(m.residual(x_a, x_v), fresh.residual(x_a, x_v)):
                assert torch.equal(a, b), name


# too few channels or nodes for the layer, axes in another order: refused, as by the module's separate operations
@pytest.mark.parametrize("a,v", [((2, 17, 16), (2, 17, 32, 3)), ((2, 17, 32), (2, 17, 16, 3)), ((2, 17, 32), (2, 16, 32, 3)),
                                 ((2, 17, 32), (17, 2, 32, 3)), ((2, 17, 32), (2, 17, 3, 32))])
def test_painn_update_refuses_what_does_not_fit(a, v):
    from ld_b200 import ops, painn
    m = painn.Update(32).cuda()
    with torch.no_grad(), pytest.raises(RuntimeError):
        m.residual(torch.zeros(a).cuda(), torch.zeros(v).cuda())
    y, row = torch.zeros(34, 96, 3).cuda(), torch.zeros(34, 32).cuda()
    with pytest.raises(RuntimeError):
        ops.painn_update_front(y, row[:33], 34, 32)
    with pytest.raises(RuntimeError):
        ops.painn_update_back(y, row, row, row, y[:, :32].contiguous(), 34, 32)


@pytest.mark.parametrize("grad", [False, True])
def test_hooks_of_the_update_run_inside_a_block(grad):
    """forward and pre-forward hooks of Update and of its parts see the calls that they saw, and what they return counts"""
    from ld_b200 import painn
    from ld_b200.graph_layers import Graph
    torch.manual_seed(6)
    block = painn.Block(3.0, 32).cuda()
    pos = torch.cumsum(torch.randn(2, 20, 3) / 3 ** 0.5, dim=1).cuda()
    graph, bonds = Graph.radius_graph(3.0, None, pos), painn.chain_bond_graph(2, 20, "cuda")
    flat = pos.reshape(-1, 3)
    x = torch.randn(2, 20, 32).cuda(), torch.randn(2, 20, 32, 3).cuda()

    def run():
        with torch.set_grad_enabled(grad):
            return [t.detach() for t in block((pos, graph, graph.rij, bonds, flat[bonds.dst] - flat[bonds.src], *x, None))[5:7]]

    plain = run()
    for name in ("", "lin_l", "lin_r", "lin_v", "mlp", "gn"):
        part = block.update.get_submodule(name)
        calls = []
        handles = [part.register_forward_pre_hook(lambda m, a: calls.append(a[0].shape)),
                   part.register_forward_hook(lambda m, a, out: calls.append(type(out)))]
        # the fused and the separate form differ by roundings
        assert all(float((a - b).norm()) <= 1e-5 * float(b.norm()) for a, b in zip(run(), plain)) and len(calls) == 2, name
        assert calls[0] == (x[1] if name.startswith("lin") else torch.empty(2, 20, 64) if name == "mlp" else x[0]).shape, name
        handles.append(part.register_forward_hook(lambda m, a, out: tuple(2 * t for t in out) if isinstance(out, tuple) else 2 * out))
        assert not all(float((a - b).norm()) <= 1e-2 * float(b.norm()) for a, b in zip(run(), plain)), name
        for h in handles:
            h.remove()
        assert all(torch.equal(a, b) for a, b in zip(run(), plain)), name


@pytest.mark.parametrize("rows", [3, 700, 1300])
def test_mlp_rows_takes_a_direct_weight_of_any_alignment(rows):
    from ld_b200 import ops
    torch.manual_seed(rows)
    mlp = ops.PackedMLP([torch.nn.Linear(a, 40).cuda() for a in (12, 40, 40)], torch.nn.Linear(12, 40, bias=False).cuda())
    x = torch.randn(rows, 12).cuda()
    want = ops.mlp3_rows(x, mlp)
    shifted = torch.empty(12 * 40 + 1, device="cuda")[1:].reshape(12, 40)
    mlp.Wdt = shifted.copy_(mlp.Wdt)
    assert shifted.data_ptr() % 16 == 4
    assert torch.equal(ops.mlp3_rows(x, mlp), want)


def _uneven(lin, kind):
    """hidden channels of layers lin[0] and lin[1] far larger or smaller than their neighbours, the same function of the inputs up
    to the activation"""
    g = torch.Generator().manual_seed(11)
    with torch.no_grad():
        for a, b in zip(lin, lin[1:]):
            if kind == "spread":      # over six orders of magnitude
                s = 10.0 ** (6 * torch.rand(a.weight.shape[0], generator=g) - 3)
            elif kind == "unit":      # one channel 1e5 in, 1e-5 out
                s = torch.ones(a.weight.shape[0])
                s[3] = 1e5
            elif kind == "off":       # one channel that its bias keeps off
                a.bias[5] = -1e6
                continue
            else:
                continue
            a.weight *= s[:, None]
            a.bias *= s
            b.weight /= s


@pytest.mark.parametrize("n,n_rbf", [(32, 9), (64, 64), (128, 8)])
@pytest.mark.parametrize("kind", ["even", "spread", "unit", "off"])
def test_split_message_with_uneven_channels(n, n_rbf, kind):
    """every channel has scales of its own: no further from 64 bits than the FP32 FMA kernel, whatever its neighbours' sizes"""
    import ctypes
    from ld_b200 import ops
    from ld_b200._lib import lib, check, ptr, stream_ptr
    g = torch.Generator().manual_seed(n)
    Nt, deg = 23, 17
    E = Nt * deg
    row_ptr = torch.arange(0, E + 1, deg).int()
    dst, rij = torch.randint(0, Nt, (E,), generator=g).int(), torch.randn(E, 3, generator=g) * 1.3
    torch.manual_seed(n)
    lin = [torch.nn.Linear(k, 4 * n) for k in (n_rbf, 4 * n, 4 * n)]
    _uneven(lin, kind)
    actv, x_v = torch.randn(Nt, 4 * n, generator=g), torch.randn(Nt, n, 3, generator=g)
    want = _message64(row_ptr, dst, rij, [(l.weight.detach(), l.bias.detach()) for l in lin], actv, x_v, 1, n_rbf, 4.0)
    mlp = ops.PackedMLP([l.cuda() for l in lin])
    args = [t.cuda() for t in (row_ptr, dst, rij)]
    actv, x_v = actv.cuda(), x_v.cuda()
    split = ops.painn_message_f32(*args, mlp, actv, x_v, 4.0, radial_kind=1)
    assert mlp._split and int(ops.tc_status(actv.device)) == 0
    fma = torch.empty(Nt, n, device="cuda"), torch.empty(Nt, n, 3, device="cuda")
    check(lib().ld_painn_message_f32(*[ptr(a) for a in args], Nt, n, n_rbf, 1, ctypes.c_float(4.0), ctypes.c_float(0.1), ptr(mlp.Wt[0]),
                                     ptr(mlp.b[0]), ptr(mlp.Wt[1]), ptr(mlp.b[1]), ptr(mlp.Wt[2]), ptr(mlp.b[2]), ptr(actv), ptr(x_v), None,
                                     None, ptr(fma[0]), ptr(fma[1]), None, stream_ptr()))
    for w, a, b in zip(want, split, fma):
        off = lambda t: float((t.cpu().double() - w).norm())  # noqa: E731
        assert off(a) <= 1.2 * off(b) + U * float(w.norm()), (off(a) / float(w.norm()), off(b) / float(w.norm()))


@pytest.mark.parametrize("chan,dim_a", [(128, 128), (64, 64), (128, 64)])
@pytest.mark.parametrize("kind", ["even", "spread", "unit", "off"])
@pytest.mark.parametrize("size", [1e-3, 1.0, 1e3])
def test_split_scalar_channel_with_uneven_channels(chan, dim_a, kind, size):
    """as above, for the l<=2 layer's scalar channel; the sizes of the features move the biases against the products"""
    from ld_b200 import bee, ops
    from ld_b200.graph_layers import Graph
    from ld_b200._lib import lib, check, ptr, stream_ptr
    g = torch.Generator().manual_seed(chan + dim_a)
    Nt, deg = 23, 13
    src, dst = torch.arange(Nt).repeat_interleave(deg), torch.randint(0, Nt, (Nt * deg,), generator=g)
    rij = torch.randn(Nt * deg, 3, generator=g) * 1.5
    torch.manual_seed(3)
    m = bee.Messages(5.0, dim_a, 32, 32, chan)
    _uneven([m.mlp_a.layers[k] for k in (0, 2, 4)], kind)
    if kind == "spread":   # psi as well
        with torch.no_grad():
            s = 10.0 ** (6 * torch.rand(dim_a, generator=g) - 3)
            for k in ("000", "110", "220"):
                getattr(m, f"Y_{k}").W *= s[:, None]
            m.mlp_a.layers[0].weight /= s
            m.mlp_a.lin_direct.weight /= s
    if kind == "off":   # the leaky slope lets a tenth of it through: as large as the others after the next weights
        with torch.no_grad():
            m.mlp_a.layers[2].weight[:, 5] *= 1e-5
            m.mlp_a.layers[4].weight[:, 5] *= 1e-5
    m = m.cuda()
    rows = torch.randn(Nt, 13, chan, generator=g) * size
    graph = Graph(src.cuda(), dst.cuda(), None, 1, Nt)
    with torch.no_grad():
        w = m._pack()
    r13, rc = rows.cuda(), rij.cuda()
    l = [r13[:, 0].contiguous(), r13[:, 1:4].transpose(1, 2).contiguous(), r13[:, 4:].transpose(1, 2).contiguous()]
    split, fma = torch.empty(Nt, dim_a, device="cuda"), torch.empty(Nt, dim_a, device="cuda")
    geo = (ptr(graph.row_ptr), ptr(graph.dst32), ptr(rc), Nt, chan, dim_a, 5.0)
    enc = (ptr(w["enc_w"]), ptr(w["enc_b"]), ptr(w["jac"]))
    check(lib().ld_bee_messages_scalar_f32_split(*geo, ptr(r13), *enc, ptr(w["split"]), None, ptr(w["b1"]), ptr(w["b2"]), ptr(w["b3"]), 0.1,
                                                 ptr(split), ptr(ops.tc_status(r13.device)), stream_ptr()))
    check(lib().ld_bee_messages_scalar_f32(*geo, *[ptr(t) for t in l], *enc, ptr(w["Yt"]), ptr(w["W1t"]), ptr(w["b1"]), ptr(w["W2t"]),
                                           ptr(w["b2"]), ptr(w["W3t"]), ptr(w["b3"]), ptr(w["Wdt"]), 0.1, ptr(fma), stream_ptr()))
    assert int(ops.tc_status(r13.device)) == 0
    p = {k: v.detach().cpu().double() for k, v in m.state_dict().items()}
    r = rij.double()
    phi = bee.radial_encode_8(r, 5.0) @ p["lin_enc.weight"].t() + p["lin_enc.bias"]
    u = r * 1.4
    u = u / torch.sqrt(1 + (u ** 2).sum(-1, keepdim=True))
    f = rows.double()[dst]
    y = [f[:, 0] * phi, torch.einsum("ekc,ek->ec", f[:, 1:4], u) * phi,
         torch.einsum("exyc,ex,ey->ec", f[:, 4:].reshape(-1, 3, 3, chan), u, u) * phi]
    psi = sum(t @ p[f"Y_{k}.W"].t() for t, k in zip(y, ("000", "110", "220")))
    h, terms = psi, psi.abs() @ p["mlp_a.lin_direct.weight"].abs().t() + psi.abs()
    for k in (0, 2, 4):
        last = h.abs()
        h = h @ p[f"mlp_a.layers.{k}.weight"].t() + p[f"mlp_a.layers.{k}.bias"]
        h = torch.nn.functional.leaky_relu(h, 0.1) if k < 4 else h
    terms += last @ p["mlp_a.layers.4.weight"].abs().t() + p["mlp_a.layers.4.bias"].abs()
    add = lambda t: torch.zeros(Nt, dim_a, dtype=torch.float64).index_add(0, src, 0.1 * t)  # noqa: E731
    want, size = add(psi + psi @ p["mlp_a.lin_direct.weight"].t() + h), add(terms)
    # per channel (their sizes differ by orders of magnitude). Both operands of a product are held to 2^-23 of their own size or
    # better, so that the last layer's products are off by 4 U at most where one term outweighs the others (the FMA kernel: U)
    a, b = ((t.cpu().double() - want).norm(dim=0) for t in (split, fma))
    assert bool((a <= 1.5 * b + 4 * U * size.norm(dim=0)).all()), float((a / (b + U * size.norm(dim=0))).max())


# many particles in a cell: all of them sorted by (cell, index) instead of ranked by counting, in blocks of 256 and 1024 threads
# and at counts that are no powers of two
@pytest.mark.parametrize("batch,nodes,box,cutoff,scale", [(2, 3001, (7.0, 7.1, 7.2), 2.3, 1.0), (1, 1500, None, 1.0, 0.02), (3, 300, None, 3.0, 0.01),
                                                         (2, 512, None, 0.5, 0.05), (1, 129, None, 3.0, 0.0), (1, 2500, None, 2.0, 0.25)])
def test_radius_graph_of_dense_systems(batch, nodes, box, cutoff, scale):
    from ld_b200 import graph as G
    from oracle import reference_math as R
    g = torch.Generator().manual_seed(nodes)
    pos = torch.rand(batch, nodes, 3, generator=g) * torch.tensor(box) if box else \
        scale * torch.cumsum(torch.randn(batch, nodes, 3, generator=g) / 3 ** 0.5, dim=1)
    b = G.RadiusGraphBuilder(batch, nodes, cutoff, box)
    got = b.build(pos.cuda())
    assert int(b.status) == 0
    oracle = R.radius_graph(pos, cutoff, box)
    key = lambda s, d: s.cpu().long() * (batch * nodes) + d.cpu().long()  # noqa: E731
    mine, want = key(got["src"], got["dst"]), key(oracle["src"], oracle["dst"])
    assert torch.equal(mine.sort().values, want.sort().values)
    assert torch.equal(got["rij"].cpu()[mine.argsort()], oracle["rij"][want.argsort()])
    # a node's neighbours come cell by cell and ascend inside a cell: at most as many descents as there are cells around it
    s, d = got["src"].long(), got["dst"].long()
    down = (s[1:] == s[:-1]) & (d[1:] < d[:-1])
    assert int(torch.bincount(s[1:][down], minlength=batch * nodes).max()) <= 27
    if scale in (0.0, 0.01):   # one cell
        assert not bool(down.any())


# the tiles between the large and the small ones, rows that 16-byte stores do not fit, in every tile
@pytest.mark.parametrize("inds,rows,dim_in,dim_out", [(0, 5000, 20, 100), (0, 4801, 9, 128), (0, 20001, 12, 127), (1, 3000, 33, 127), (1, 2999, 18, 68),
                                                      (1, 5001, 6, 129), (2, 1500, 18, 65), (2, 2047, 10, 128), (2, 2500, 5, 126), (2, 40, 8, 7)])
def test_tensor_linear_middle_tiles_and_ragged_rows(inds, rows, dim_in, dim_out):
    from ld_b200 import ops
    g = torch.Generator().manual_seed(rows)
    W, x = torch.randn(dim_out, dim_in, generator=g), torch.randn(rows, dim_in, *[3] * inds, generator=g)
    bound = dim_in * U * _linear64(W.abs(), x.abs(), inds)   # n products in any order, with FMAs
    guard = torch.full((rows * dim_out * 3 ** inds + 64,), 7.0, device="cuda")
    from ld_b200._lib import lib, check, ptr, stream_ptr
    Wc, xc = W.cuda(), x.cuda()
    for shift in (0, 1):   # an output that starts at no 16-byte boundary
        out = guard[shift: rows * dim_out * 3 ** inds + shift].reshape(rows, dim_out, *[3] * inds)
        check(lib().ld_tensor_linear(inds, ptr(Wc), dim_in, 1, ptr(xc), out.data_ptr(), rows, dim_in, dim_out, stream_ptr()))
        assert bool(((out.cpu().double() - _linear64(W, x, inds)).abs() <= bound).all())
        assert bool((guard[rows * dim_out * 3 ** inds + shift:] == 7.0).all())
        guard.fill_(7.0)


def _chunk_graph(nodes, chunk, seed):
    """0 to 3 edges a node, whose ends lie in the same chunk of nodes; one stretch without edges, one node with many"""
    g = torch.Generator().manual_seed(seed)
    deg = torch.randint(0, 4, (nodes,), generator=g)
    deg[nodes // 3: nodes // 3 + chunk // 2] = 0
    deg[nodes // 2] = 300
    src = torch.repeat_interleave(torch.arange(nodes), deg)
    lo = src // chunk * chunk
    dst = lo + (torch.rand(len(src), generator=g) * (torch.clamp(lo + chunk, max=nodes) - lo)).long()
    return deg, src, dst, torch.randn(len(src), 3, generator=g) * 1.3


# the blocks walk the nodes in segments of about 40 MB of gathered rows (11.7 k nodes at n = 128): rings, accumulators and sums go
# on from one segment to the next, blocks have no edges in some of them
@pytest.mark.parametrize("n,nodes", [(32, 100_000), (64, 52_000), (128, 26_000)])
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_messages_over_several_segments(n, nodes, precision):
    """the whole graph against its chunks of less than one segment, computed by themselves: the same bits"""
    from ld_b200 import ops
    chunk = 5000
    deg, src, dst, rij = _chunk_graph(nodes, chunk, n)
    torch.manual_seed(n)
    mlp = ops.PackedMLP([torch.nn.Linear(k, 4 * n).cuda() for k in (8, 4 * n, 4 * n)])
    fused = ops.painn_message_bf16_tc if precision == "bf16" else ops.painn_message_f32
    actv, x_v, res_a = torch.randn(nodes, 4 * n, device="cuda"), torch.randn(nodes, n, 3, device="cuda"), torch.randn(nodes, n, device="cuda")
    row_ptr = torch.cat([torch.zeros(1, dtype=torch.long), deg.cumsum(0)])

    def run(lo, hi, residual):
        e = slice(int(row_ptr[lo]), int(row_ptr[hi]))
        return fused((row_ptr[lo:hi + 1] - row_ptr[lo]).int().cuda(), (dst[e] - lo).int().cuda(), rij[e].cuda(), mlp, actv[lo:hi], x_v[lo:hi], 4.0,
                     radial_kind=1, res_a=res_a[lo:hi] if residual else None, res_v=x_v[lo:hi] if residual else None)

    for residual in (False, True):
        whole = run(0, nodes, residual)
        for lo in range(0, nodes, chunk):
            for w, p in zip(whole, run(lo, min(lo + chunk, nodes), residual)):
                assert torch.equal(w[lo:lo + chunk], p), lo
    assert bool((run(0, nodes, False)[0][deg == 0] == 0).all()) and int(ops.tc_status("cuda")) == 0


@pytest.mark.parametrize("chan,dim_a,nodes", [(128, 128, 20_000), (64, 64, 40_000), (128, 64, 20_000), (64, 128, 40_000)])
def test_scalar_channel_over_several_segments(chan, dim_a, nodes):
    from ld_b200 import bee, ops
    from ld_b200._lib import lib, check, ptr, stream_ptr
    chunk = 5000
    deg, src, dst, rij = _chunk_graph(nodes, chunk, chan)
    torch.manual_seed(chan)
    m = bee.Messages(5.0, dim_a, 32, 32, chan).cuda()
    with torch.no_grad():
        w = m._pack()
    rows = torch.randn(nodes, 13, chan, device="cuda")
    row_ptr = torch.cat([torch.zeros(1, dtype=torch.long), deg.cumsum(0)])

    def run(lo, hi):
        e = slice(int(row_ptr[lo]), int(row_ptr[hi]))
        rp, d, r, part = (row_ptr[lo:hi + 1] - row_ptr[lo]).int().cuda(), (dst[e] - lo).int().cuda(), rij[e].cuda(), rows[lo:hi]
        out = torch.full((hi - lo, dim_a), 7.0, device="cuda")
        check(lib().ld_bee_messages_scalar_f32_split(ptr(rp), ptr(d), ptr(r), hi - lo, chan, dim_a, 5.0, ptr(part), ptr(w["enc_w"]), ptr(w["enc_b"]),
                                                     ptr(w["jac"]), ptr(w["split"]), None, ptr(w["b1"]), ptr(w["b2"]), ptr(w["b3"]), 0.1, ptr(out),
                                                     ptr(ops.tc_status("cuda")), stream_ptr()))
        return out

    whole = run(0, nodes)
    for lo in range(0, nodes, chunk):
        assert torch.equal(whole[lo:lo + chunk], run(lo, min(lo + chunk, nodes))), lo
    assert bool((whole[deg == 0] == 0).all()) and int(ops.tc_status("cuda")) == 0


@pytest.mark.parametrize("kernel", ["f32-32", "f32-64", "f32-128", "bf16-32", "bf16-64", "bf16-128", "scalar-64-64", "scalar-128-128"])
def test_edge_kernels_repeat_themselves(kernel):
    """a slab that is read before it has landed, or a plane that is still being written, would show as bits that differ from one
    launch to the next: a few tiles a block, 600 launches"""
    from ld_b200 import bee, ops
    from ld_b200._lib import lib, check, ptr, stream_ptr
    kind, n = kernel.split("-")[0], int(kernel.split("-")[1])
    deg, src, dst, rij = _chunk_graph(9000, 9000, 3)
    row_ptr = torch.cat([torch.zeros(1, dtype=torch.long), deg.cumsum(0)]).int().cuda()
    dst, rij, nodes = dst.int().cuda(), rij.cuda(), len(deg)
    torch.manual_seed(n)
    if kind == "scalar":
        m = bee.Messages(5.0, n, 32, 32, n).cuda()
        with torch.no_grad():
            w = m._pack()
        rows = torch.randn(nodes, 13, n, device="cuda")

        def run():
            out = torch.empty(nodes, n, device="cuda")
            check(lib().ld_bee_messages_scalar_f32_split(ptr(row_ptr), ptr(dst), ptr(rij), nodes, n, n, 5.0, ptr(rows), ptr(w["enc_w"]),
                                                         ptr(w["enc_b"]), ptr(w["jac"]), ptr(w["split"]), None, ptr(w["b1"]), ptr(w["b2"]),
                                                         ptr(w["b3"]), 0.1, ptr(out), ptr(ops.tc_status("cuda")), stream_ptr()))
            return (out,)
    else:
        mlp = ops.PackedMLP([torch.nn.Linear(k, 4 * n).cuda() for k in (8, 4 * n, 4 * n)])
        actv, x_v = torch.randn(nodes, 4 * n, device="cuda"), torch.randn(nodes, n, 3, device="cuda")
        fused = ops.painn_message_bf16_tc if kind == "bf16" else ops.painn_message_f32
        run = lambda: fused(row_ptr, dst, rij, mlp, actv, x_v, 4.0, radial_kind=1)  # noqa: E731
    first, other = run(), torch.zeros((), dtype=torch.bool, device="cuda")
    for _ in range(600):
        for a, b in zip(first, run()):
            other |= (a != b).any()
    assert not bool(other) and int(ops.tc_status("cuda")) == 0


def test_painn_update_refuses_weights_that_are_elsewhere():
    """weights in host memory are refused, weights that are not contiguous float32 take the separate operations"""
    from ld_b200 import painn
    torch.manual_seed(8)
    x_a, x_v = torch.randn(2, 5, 32).cuda(), torch.randn(2, 5, 32, 3).cuda()
    with torch.no_grad(), pytest.raises(RuntimeError):
        painn.Update(32).residual(x_a, x_v)
    m = painn.Update(32).cuda()
    with torch.no_grad():
        want = m.residual(x_a, x_v)
        m.lin_v.W.data = m.lin_v.W.data.t().contiguous().t()
        got = m.residual(x_a, x_v)
    assert not m.lin_v.W.is_contiguous()
    assert all(float((a - b).norm()) <= 1e-5 * float(b.norm()) for a, b in zip(got, want))


# tiles of 32, 64 and 128 outputs that lie in one of the three matrices, that straddle two, that hold all three
@pytest.mark.parametrize("n,rows", [(4, 100), (24, 6000), (32, 37), (40, 5001), (64, 2500), (64, 6000), (100, 3000), (128, 37), (128, 3000), (128, 6001)])
def test_update_mix_equals_the_stacked_mixing(n, rows):
    from ld_b200 import ops
    torch.manual_seed(n)
    W = [torch.randn(n, n).cuda() for _ in range(3)]
    x = torch.randn(rows, n, 3).cuda()
    assert torch.equal(ops.painn_update_mix(*W, x, rows, n), ops.tensor_linear_fwd(1, torch.cat(W), x))
