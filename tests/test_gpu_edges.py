"""Sizes at the edges of the tiles and of the dispatch rules of single kernels, against the CPU checker: rows of every remainder
modulo the access width, planes and tensors on either side of a rule's limit, buffers off their usual alignment."""
import collections
import types

import numpy as np
import pytest

import synth
from util import assert_bits_equal

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def capi():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import nnforge_b200.capi as capi
    return capi


@pytest.fixture
def tuning(capi):
    yield capi.set_tuning
    capi.set_tuning("reset", 0)


def dev(a, offset=0):
    """A CUDA copy of the array, `offset` floats behind an aligned address."""
    t = torch.empty(a.size + offset, dtype=torch.float32 if a.dtype == np.float32 else torch.int32, device="cuda")
    t[offset:].copy_(torch.from_numpy(np.ascontiguousarray(a)).reshape(-1))
    return t[offset:].view(a.shape)


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


def launches(call):
    """What the call puts on its stream, from a capture of it: the CTAs per cluster of each kernel (1: no cluster), "memset", or "other".
    The call itself is not run."""
    import ctypes as ct
    cuda = ct.CDLL("libcuda.so.1")

    def ok(status):
        assert status == 0, "status %d" % status

    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    handle, count = ct.c_void_p(graph.raw_cuda_graph()), ct.c_size_t(0)
    ok(cuda.cuGraphGetNodes(handle, None, ct.byref(count)))
    nodes = (ct.c_void_p * count.value)()
    ok(cuda.cuGraphGetNodes(handle, nodes, ct.byref(count)))
    out = []
    for node in nodes:
        kind, value = ct.c_int(), (ct.c_uint32 * 16)()
        ok(cuda.cuGraphNodeGetType(ct.c_void_p(node), ct.byref(kind)))
        if kind.value == 0:         # CU_GRAPH_NODE_TYPE_KERNEL, CU_LAUNCH_ATTRIBUTE_CLUSTER_DIMENSION
            ok(cuda.cuGraphKernelNodeGetAttribute(ct.c_void_p(node), 4, value))
        out.append({0: max(1, value[0]), 2: "memset"}.get(kind.value, "other"))
    return out


# widths of every remainder modulo 4 up to more columns than a warp serves; heights of one pair of rows up to several, odd and even
ROW_SHAPES = [(2, 3, 3, 3), (1, 5, 4, 4), (3, 2, 5, 5), (2, 2, 6, 6), (2, 3, 7, 7), (1, 3, 8, 9), (2, 1, 9, 34), (1, 2, 3, 131), (1, 1, 10, 130), (1, 1, 11, 128),
              (5, 7, 13, 13), (2, 3, 33, 35), (9, 16, 14, 14)]


@pytest.mark.parametrize("shape", ROW_SHAPES)
@pytest.mark.parametrize("win", [2, 3])
@pytest.mark.parametrize("round_up", [False, True])
@pytest.mark.parametrize("staged", [0, 1])
def test_max_subsampling_rows_and_plane_groups(capi, oracle, tuning, shape, win, round_up, staged):
    """3x3 and 2x2 windows at stride 2 through the row kernels and through the plane-group kernels that large tensors take, with
    NaNs and infinities among the values, stand-alone and fused, in place, and with buffers that only allow narrower accesses."""
    tuning("pool_staged", staged)
    g = synth.rng(3, salt=sum(shape) * 7 + win)
    n, c = shape[:2]
    ru = (round_up, round_up)
    x = synth.with_edges(g, np.maximum(synth.normal(g, shape), 0))
    x.reshape(-1)[g.choice(x.size, max(1, x.size // 40), replace=False)] = np.nan
    for offset in (0, 2, 1):
        for is_min in (False, True):
            p = capi.pool((win, win), (2, 2), ru, is_min)
            want, want_idx = oracle.maxpool_fwd(x, (win, win), (2, 2), ru, is_min)
            y, idx = torch.empty(want.shape, device="cuda"), torch.zeros(want.shape, dtype=torch.int32, device="cuda")
            capi.maxpool_fwd(y, idx, dev(x, offset), p)
            assert_bits_equal(host(idx).view(np.uint32), want_idx, "argmax")
            assert_bits_equal(host(y), want, "values")
        dy, dx0 = synth.normal(g, want.shape), synth.normal(g, shape)
        dx = dev(dx0, offset)
        capi.maxpool_bwd(dx, dev(dy), idx, p)
        assert_bits_equal(host(dx), oracle.maxpool_bwd(dy, want_idx, shape), "gradient")
        dx = dev(dx0, offset)
        capi.maxpool_bwd(dx, dev(dy), idx, p, add_to_destination=True)
        assert_bits_equal(host(dx), oracle.maxpool_bwd(dy, want_idx, shape, dx=dx0), "gradient accumulated")

    x, r = synth.normal(g, shape), synth.normal(g, shape)
    bn = synth.bn_params(g, c)
    p = capi.pool((win, win), (2, 2), ru)
    bnd = [dev(a) for a in bn]
    s = oracle.add_fwd([oracle.bn_infer(x, *bn), r], 1.0)
    z_want = oracle.relu_fwd(s, 0.0)
    want, want_idx = oracle.maxpool_fwd(z_want, (win, win), (2, 2), ru)
    dyp = synth.normal(g, want.shape)
    ds = oracle.relu_bwd(oracle.maxpool_bwd(dyp, want_idx, shape), s, 0.0)
    dx_want = (ds * (bn[0] * bn[3]).astype(np.float32)[None, :, None, None]).astype(np.float32)
    for offset, over in ((0, None), (2, None), (1, None), (0, "x"), (1, "residual")):
        xd, rd = dev(x, offset), dev(r, offset)
        z = {"x": xd, "residual": rd}.get(over, torch.empty(x.size + offset, device="cuda")[offset:].view(shape))
        y, idx = torch.empty(want.shape, device="cuda"), torch.zeros(want.shape, dtype=torch.int32, device="cuda")
        capi.bn_add_relu_maxpool_fwd(z, y, idx, xd, rd, bnd, 0.0, p)
        assert_bits_equal(host(z), z_want, "z")
        assert_bits_equal(host(y), want, "pooled")
        assert_bits_equal(host(idx).view(np.uint32), want_idx, "fused argmax")
        dx, dr = dev(np.zeros(shape, np.float32), offset), dev(np.zeros(shape, np.float32), offset)
        capi.bn_add_relu_maxpool_bwd(dx, dr, dev(dyp), idx, z, bnd[0], bnd[3], 0.0, p)
        assert_bits_equal(host(dr), ds, "dresidual")
        assert_bits_equal(host(dx), dx_want, "dx")


# values on either side of the limits beyond which plane groups take small planes
@pytest.mark.parametrize("plane,win,million", [((9, 9), 3, 2.5), ((13, 13), 3, 5), ((21, 21), 3, 15), ((6, 6), 3, 4), ((10, 10), 3, 12), ((14, 14), 3, 20), ((9, 9), 2, 6), ((5, 5), 2, 2),
                                               ((21, 21), 2, 16), ((6, 6), 2, 35), ((4, 4), 3, 18), ((4, 4), 2, 18), ((7, 7), 2, 7.5), ((11, 11), 2, 7.5), ((20, 4), 3, 4.5), ((20, 4), 2, 4.5)])
@pytest.mark.parametrize("offset", [0, 1])
def test_max_subsampling_of_many_small_planes(capi, tuning, plane, win, million, offset):
    """Whichever kernels take the layer, and behind the fused layers where rows are 4 wide, the results are those of the plane-group kernels."""
    hw = plane[0] * plane[1]
    p = capi.pool((win, win), (2, 2))
    for planes in (int(million * 1e6 / hw) - 1, int(million * 1e6 / hw) + 3):
        shape = (planes, 1) + plane
        x = torch.empty(planes * hw + offset, device="cuda").normal_()[offset:].view(shape)
        out = (planes, 1) + capi.pool_out_shape(plane[0], plane[1], p)
        got = []
        for staged in (0, 1):
            tuning("pool_staged", staged)
            y, idx = torch.full(out, float("nan"), device="cuda"), torch.zeros(out, dtype=torch.int32, device="cuda")
            dx = torch.full_like(x, float("nan"))
            capi.maxpool_fwd(y, idx, x, p)
            capi.maxpool_bwd(dx, y, idx, p)
            got.append([y, idx, dx])
            if plane[1] == 4:
                one, zero = torch.ones(1, device="cuda"), torch.zeros(1, device="cuda")
                z, dr = torch.empty_like(x), torch.full_like(x, float("nan"))
                capi.bn_add_relu_maxpool_fwd(z, y, idx, x, x, (one * 1.5, one, zero, one), 0.0, p)
                capi.bn_add_relu_maxpool_bwd(dx, dr, y, idx, z, one * 1.5, one, 0.0, p)
                got[-1] += [z, dr, dx]
        for a, b in zip(*got):
            assert torch.equal(a, b)


@pytest.mark.parametrize("win", [2, 3])
def test_fused_max_subsampling_of_planes_beyond_shared_memory(capi, oracle, win):
    """Planes of 231 KB: taken at stride 2 where z is written to a buffer of its own, refused over x, over the residual and at other
    strides, as the header says."""
    g = synth.rng(3, salt=win)
    shape = (1, 2, 241, 246)
    x, r = synth.normal(g, shape), synth.normal(g, shape)
    bn = synth.bn_params(g, 2)
    bnd, xd, rd = [dev(a) for a in bn], dev(x), dev(r)
    z_want = oracle.relu_fwd(oracle.add_fwd([oracle.bn_infer(x, *bn), r], 1.0), 0.0)
    want, want_idx = oracle.maxpool_fwd(z_want, (win, win), (2, 2), (False, False))
    p = capi.pool((win, win), (2, 2))
    z, y, idx = torch.empty(shape, device="cuda"), torch.empty(want.shape, device="cuda"), torch.zeros(want.shape, dtype=torch.int32, device="cuda")
    capi.bn_add_relu_maxpool_fwd(z, y, idx, xd, rd, bnd, 0.0, p)
    assert_bits_equal(host(z), z_want, "z")
    assert_bits_equal(host(y), want, "pooled")
    assert_bits_equal(host(idx).view(np.uint32), want_idx, "argmax")
    for over in (xd, rd):
        with pytest.raises(capi.NnfError, match="does not fit"):
            capi.bn_add_relu_maxpool_fwd(over, y, idx, xd, rd, bnd, 0.0, p)
    with pytest.raises(capi.NnfError, match="does not fit"):
        capi.bn_add_relu_maxpool_fwd(z, y, idx, xd, rd, bnd, 0.0, capi.pool((win, win), (1, 1)))


@pytest.mark.parametrize("kind", ["none", "vanilla", "nesterov", "adam"])
@pytest.mark.parametrize("chunks", [1, 48, 49, 160, 161, 500, 501])
def test_optimiser_step_chunk_counts_and_alignment(capi, oracle, kind, chunks):
    """Chunk counts on either side of the parameter blocks' capacities; chunks of every remainder modulo a thread's four weights and a
    CTA's 1024, each with its buffers aligned and one float off."""
    g = synth.rng(1, salt=8100 + chunks)
    mtype = {"none": capi.MOMENTUM_NONE, "vanilla": capi.MOMENTUM_VANILLA, "nesterov": capi.MOMENTUM_NESTEROV, "adam": capi.MOMENTUM_ADAM}[kind]
    sizes = [1023, 1024, 1025, 1, 2, 3, 4, 5, 2047, 2050]
    names = ["data", "gradient"] + (["prev_upd"] if kind != "none" else []) + (["prev_upd2"] if kind == "adam" else [])
    hostp, devp = [], []
    for k in range(chunks):
        n = sizes[k % len(sizes)]
        hp = {"data": synth.normal(g, (n,)), "gradient": synth.normal(g, (n,)), "prev_upd": synth.normal(g, (n,), 0.0, 0.01),
              "prev_upd2": np.abs(synth.normal(g, (n,), 0.0, 0.1))}
        dp = {name: dev(hp[name], (k // len(sizes)) % 2 if name != "gradient" else 0) for name in names}
        dp.update(learning_rate=0.01, weight_decay=0.0005 if k % 2 else 0.0, update_accum=torch.zeros(1, dtype=torch.float64, device="cuda"))
        hostp.append(hp)
        devp.append(dp)
    capi.apply_gradient(devp, mtype, 0.9, 0.999, 1.0 / 32, 2)
    for k, (hp, dp) in enumerate(zip(hostp, devp)):
        accum = oracle.apply_gradient(hp["data"], hp["gradient"], hp["prev_upd"], hp["prev_upd2"], kind, 0.01, 1.0 / 32, dp["weight_decay"], 0.9, 0.999, 2)
        assert not host(dp["gradient"]).any()
        for name in names:
            if name != "gradient":
                assert_bits_equal(host(dp[name]), hp[name], "%s, chunk %d" % (name, k))
        # two orders of a double sum of at most 2050 terms of one sign: 2050 * 2^-53 < 3e-13 relative
        assert abs(float(host(dp["update_accum"])[0]) - accum) <= 1e-12 * accum


def test_optimiser_step_chunks_of_any_mapping(capi):
    """The same step from plain dicts and from other mappings, optional fields there, absent and None."""
    def chunks(kind):
        g = torch.Generator(device="cuda")
        g.manual_seed(12)
        make = lambda: torch.empty(70, device="cuda").normal_(generator=g)
        return [kind(data=make(), gradient=make(), prev_upd=make(), prev_upd2=None, update_accum=torch.zeros(1, dtype=torch.float64, device="cuda"),
                     learning_rate=0.1, weight_decay=0.01), kind(data=make(), gradient=make(), prev_upd=make(), learning_rate=0.1)]

    results = []
    for kind in (dict, collections.OrderedDict, collections.UserDict, lambda **kw: types.MappingProxyType(kw)):
        parts = chunks(kind)
        capi.apply_gradient(parts, capi.MOMENTUM_VANILLA, 0.9)
        results.append([host(p[f]).copy() for p in parts for f in ("data", "gradient", "prev_upd")] + [host(parts[0]["update_accum"]).copy()])
    for got in results[1:]:
        for a, b in zip(results[0], got):
            assert a.tobytes() == b.tobytes()


def test_layer_objects_take_storages():
    """The layer objects ask a buffer for its address alone."""
    import nnforge_b200.host as host_layers
    x = torch.empty(3, 4, 5, 5, device="cuda").normal_()
    y, z = torch.empty_like(x), torch.empty_like(x)
    tester = host_layers.Tester("TanH", 4, 5, 5)
    tester.enqueue_forward_propagation(y, [], [x], 3)
    tester.enqueue_forward_propagation(z.untyped_storage(), [], [x.untyped_storage()], 3)
    assert_bits_equal(host(z), host(y), "storages")


# planes of whole float4s, planes of every remainder modulo 4, entries that do not divide by the CTAs, a tensor that ends inside a float4
TRAIN_SHAPES = [(8, 3, 8, 8), (9, 4, 9, 9), (5, 5, 9, 11), (16, 3, 13, 10), (33, 7, 27, 27), (4, 2, 56, 56), (17, 6, 19, 21), (64, 1, 8, 8), (12, 3, 55, 57),
                (7, 8, 7, 7), (5, 9, 4, 4)]


@pytest.mark.parametrize("shape", TRAIN_SHAPES)
@pytest.mark.parametrize("acts", ["none", "relu", "prelu_elu", "tanh"])
@pytest.mark.parametrize("ctas", [0, 1, 2, 4, 8])
def test_training_batch_norm_in_a_cluster(capi, tuning, shape, acts, ctas):
    """The cluster form at every count of CTAs per channel, out of place and in place, against float64 arithmetic. y and dx carry
    some ten roundings of 2^-24 and an exponential good to 2^-22: 1e-6 and 3e-6 of the 2-norm. A channel's gradient is a sum of m
    terms of either sign around 1, each good to some 2^-22: 4e-6 * sqrt(m)."""
    tuning("chain_cluster", ctas)
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(shape) * 3 + ctas)
    n, c, h, w = shape
    x = torch.empty(shape, device="cuda").normal_(0.5, 2.0, generator=g)
    dy = torch.empty(shape, device="cuda").normal_(generator=g)
    gamma = torch.empty(c, device="cuda").uniform_(0.5, 1.5, generator=g)
    beta, mean, slope = (torch.empty(c, device="cuda").normal_(0.0, 0.1, generator=g) for _ in range(3))
    slope.abs_()
    invsigma = torch.empty(c, device="cuda").uniform_(0.5, 1.5, generator=g)
    per = lambda t: t.view(1, -1, 1, 1)

    def norm(xd, ga, be):
        var, mu = torch.var_mean(xd, dim=(0, 2, 3), correction=0)
        inv = (var + 1e-5).rsqrt()
        return (xd - per(mu)) * per(inv) * per(ga) + per(be), mu, inv

    # off the rectifiers' kink, where two correct evaluations may be on different sides
    x.add_((norm(x.double(), gamma.double(), beta.double())[0].abs() < 1e-4).float() * 0.01)
    xd, sl, ga, be = (t.double().requires_grad_(True) for t in (x, slope, gamma, beta))
    u, mu, inv = norm(xd, ga, be)
    want = {"none": lambda: u, "relu": lambda: torch.relu(u), "tanh": lambda: torch.tanh(u),
            "prelu_elu": lambda: torch.nn.functional.elu(torch.where(u >= 0, u, u * per(sl)))}[acts]()
    want.backward(dy.double())
    chain = {"none": [], "relu": [capi.relu()], "prelu_elu": [capi.prelu(slope), capi.elu()], "tanh": [capi.tanh(1.0, 1.0)]}[acts]
    ws = torch.empty(capi.bn_train_workspace_bytes(n, c, h * w), dtype=torch.uint8, device="cuda")
    close = lambda a, b, tol: float((a.double() - b.detach()).norm()) <= tol * float(b.detach().norm()) + 1e-12
    room = 4e-6 * (n * h * w) ** 0.5

    def in_cluster(backward, got):
        # a CTA takes at most 220 KB of a channel's entries, 56 KB where planes are whole float4s; beyond that any other form is right
        whole = h * w % 4 == 0
        row = (h * w // 4 if whole else (h * w + 6) // 4) * 16 * (2 if backward else 1)
        if -(-n // (ctas or 8)) * row <= (56 if whole else 220) * 1024:
            assert len(got) == 1 and got[0] in ([ctas] if ctas else [1, 2, 4, 8]), got
        else:
            assert len(got) > 1, got

    for in_place in (False, True):
        y = x.clone() if in_place else torch.full_like(x, float("nan"))
        saved, sums, bsums = (torch.full((k * c,), float("nan"), device="cuda") for k in (2, 2, 3))
        forward = lambda: capi.bn_train_fwd(y, saved, sums, y if in_place else x, gamma, beta, 1e-5, chain, workspace=ws)
        in_cluster(False, launches(forward))
        forward()
        assert close(y, want, 1e-6)
        assert close(saved[:c], mu, 1e-6) and close(saved[c:], inv, 1e-6)
        assert close(sums[:c], xd.sum((0, 2, 3)), 2e-6) and close(sums[c:], (xd ** 2).sum((0, 2, 3)), 2e-6)
        grads = [torch.full((c,), 0.25, device="cuda") for _ in range(5)]
        dx = dy.clone() if in_place else torch.full_like(x, float("nan"))
        backward = lambda: capi.bn_train_bwd(dx, bsums, dx if in_place else dy, x, gamma, beta, saved, chain, grad_gamma=grads[0], grad_beta=grads[1],
                                             grad_mean=grads[2], grad_invsigma=grads[3], grad_slope=grads[4] if acts == "prelu_elu" else None, mean=mean,
                                             invsigma=invsigma, entry_count=float(n), workspace=ws)
        in_cluster(True, launches(backward))
        backward()
        assert close(dx, xd.grad, 3e-6)
        for got, gradient in ((grads[0], ga), (grads[1], be)) + (((grads[4], sl),) if acts == "prelu_elu" else ()):
            assert float((got.double() - 0.25 - gradient.grad).abs().max()) <= room
        assert close(grads[2] - 0.25, n * (saved[:c] - mean).double(), 1e-5) and close(grads[3] - 0.25, n * (saved[c:] - invsigma).double(), 1e-5)
        if h * w % 4 == 0:
            report = torch.zeros(capi.REPORT_WORDS, dtype=torch.int64).pin_memory()
            capi.read_report(report, ws)
            torch.cuda.synchronize()
            assert capi.parse_report(report)["status"] == 0


@pytest.mark.parametrize("shape", [(8, 5, 13, 13), (8, 8, 12, 12)])
@pytest.mark.parametrize("mean", [0.0, 500.0])
@pytest.mark.parametrize("outlier", [0.0, 20.0])
def test_training_batch_norm_in_a_cluster_far_from_zero(capi, shape, mean, outlier):
    """Means of 500 standard deviations and a first element, the one the sums are taken around, 20 of them from the mean. A thread adds
    the squares of at most 4 elements in float, each good to 2^-24 of (1 + outlier)^2, before sums are taken in double: half of that,
    relative, is the inverse deviation's error. y also carries the rounding of the mean times the scale, mean * 2^-23."""
    n, c, h, w = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(int(mean + outlier))
    x = torch.empty(shape, device="cuda").normal_(mean, 1.0, generator=g)
    x[0, :, 0, 0] = mean + outlier
    gamma, beta = torch.ones(c, device="cuda"), torch.zeros(c, device="cuda")
    y, saved, sums = torch.empty_like(x), torch.empty(2 * c, device="cuda"), torch.empty(2 * c, device="cuda")
    ws = torch.empty(capi.bn_train_workspace_bytes(n, c, h * w), dtype=torch.uint8, device="cuda")
    forward = lambda: capi.bn_train_fwd(y, saved, sums, x, gamma, beta, 1e-5, [], workspace=ws)
    got = launches(forward)
    assert len(got) == 1 and got[0] != "memset"
    forward()
    xd = x.double()
    var, mu = torch.var_mean(xd, dim=(0, 2, 3), correction=0)
    inv = (var + 1e-5).rsqrt()
    tol = 4 * (1 + outlier) ** 2 * 2.0 ** -25 + 2.0 ** -23
    assert float((saved[:c] - mu).abs().max()) <= 2.0 ** -23 * mean + (1 + outlier) * 2.0 ** -22
    assert float(((saved[c:] - inv) / inv).abs().max()) <= tol
    want = (xd - mu.view(1, -1, 1, 1)) * inv.view(1, -1, 1, 1)
    assert float((y - want).norm() / want.norm()) <= tol + (1 + mean) * 2.0 ** -23


@pytest.mark.parametrize("shape,clusters", [((3, 5, 3, 5), False), ((3, 5, 5, 5), True), ((3, 5, 2, 6), False), ((3, 5, 4, 4), True)])
def test_smallest_planes_of_the_cluster_form(capi, shape, clusters):
    """Planes on either side of the smallest that a cluster takes, ragged and of whole float4s."""
    n, c, h, w = shape
    x = torch.empty(shape, device="cuda").normal_()
    gamma, beta = torch.ones(c, device="cuda"), torch.zeros(c, device="cuda")
    y, saved, sums = torch.empty_like(x), torch.empty(2 * c, device="cuda"), torch.empty(2 * c, device="cuda")
    ws = torch.empty(capi.bn_train_workspace_bytes(n, c, h * w), dtype=torch.uint8, device="cuda")
    forward = lambda: capi.bn_train_fwd(y, saved, sums, x, gamma, beta, 1e-5, [], workspace=ws)
    assert (len(launches(forward)) == 1) == clusters
    forward()
    want = torch.nn.functional.batch_norm(x.double(), None, None, training=True, eps=1e-5)
    assert float((y - want).norm() / want.norm()) <= 1e-6


@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("plane,kb", [((4, 4), 56), ((7, 7), 104)])
def test_largest_slices_of_the_cluster_form(capi, tuning, plane, kb, backward):
    """As many entries as a CTA's slice may hold, and one more: 56 KB of planes of whole float4s, 104 KB of ragged ones that channel groups
    take otherwise. One CTA per channel."""
    tuning("chain_cluster", 1)
    hw = plane[0] * plane[1]
    row = (hw // 4 if hw % 4 == 0 else (hw + 6) // 4) * 16 * (2 if backward else 1)
    for n, clusters in ((kb * 1024 // row, True), (kb * 1024 // row + 1, False)):
        x, dy = (torch.empty((n, 8) + plane, device="cuda").normal_() for _ in range(2))
        gamma, beta = torch.ones(8, device="cuda"), torch.zeros(8, device="cuda")
        out, saved, sums = torch.empty_like(x), torch.empty(16, device="cuda"), torch.empty(24, device="cuda")
        ws = torch.empty(capi.bn_train_workspace_bytes(n, 8, hw), dtype=torch.uint8, device="cuda")
        xd = x.double().requires_grad_(True)
        want = torch.nn.functional.batch_norm(xd, None, None, training=True, eps=1e-5)
        forward = lambda: capi.bn_train_fwd(out, saved, sums, x, gamma, beta, 1e-5, [], workspace=ws)
        call = forward
        if backward:
            forward()
            want.backward(dy.double())
            want = xd.grad
            call = lambda: capi.bn_train_bwd(out, sums, dy, x, gamma, beta, saved, [], workspace=ws)
        assert (launches(call) == [1]) == clusters
        call()
        assert float((out - want.detach()).norm() / want.detach().norm()) <= (3e-6 if backward else 1e-6)


@pytest.mark.parametrize("shape,clusters", [((2048, 248, 7, 7), True), ((2048, 256, 7, 7), False), ((1024, 256, 9, 11), True)])
def test_small_ragged_planes_of_large_tensors(capi, shape, clusters):
    """Forward, 100 MB on either side for planes of 49 elements, and more than that for larger planes; backward, clusters throughout."""
    n, c, h, w = shape
    x, dy = (torch.empty(shape, device="cuda").normal_() for _ in range(2))
    gamma, beta = torch.ones(c, device="cuda"), torch.zeros(c, device="cuda")
    y, dx, saved, sums, bsums = torch.empty_like(x), torch.empty_like(x), *(torch.empty(k * c, device="cuda") for k in (2, 2, 3))
    ws = torch.empty(capi.bn_train_workspace_bytes(n, c, h * w), dtype=torch.uint8, device="cuda")
    forward = lambda: capi.bn_train_fwd(y, saved, sums, x, gamma, beta, 1e-5, [], workspace=ws)
    assert (len(launches(forward)) == 1) == clusters
    assert len(launches(lambda: capi.bn_train_bwd(dx, bsums, dy, x, gamma, beta, saved, [], workspace=ws))) == 1
    forward()
    want = torch.nn.functional.batch_norm(x.double(), None, None, training=True, eps=1e-5)
    assert float((y - want).norm() / want.norm()) <= 1e-6


@pytest.mark.parametrize("shape", [(49200, 4, 4, 4), (3000, 8, 3, 3), (600, 8, 28, 28)])
def test_training_batch_norm_stays_in_its_workspace(capi, tuning, shape):
    """As many items per channel as a plan makes (64 at most), with a workspace of exactly the size that is asked for: what follows it
    stays as it was."""
    tuning("chain_cluster", 99)
    tuning("chain_s_kb", 1)
    n, c, h, w = shape
    x, dy = (torch.empty(shape, device="cuda").normal_() for _ in range(2))
    gamma, beta = torch.ones(c, device="cuda"), torch.zeros(c, device="cuda")
    y, dx = torch.empty_like(x), torch.empty_like(x)
    saved, sums, bsums = (torch.empty(k * c, device="cuda") for k in (2, 2, 3))
    need = capi.bn_train_workspace_bytes(n, c, h * w)
    room = torch.full((need + 65536,), 0xa5, dtype=torch.uint8, device="cuda")
    ws = room[:need]
    capi.bn_train_fwd(y, saved, sums, x, gamma, beta, 1e-5, [], workspace=ws)
    capi.bn_train_bwd(dx, bsums, dy, x, gamma, beta, saved, [], workspace=ws)
    assert bool((room[need:] == 0xa5).all())
    xd = x.double().requires_grad_(True)
    want = torch.nn.functional.batch_norm(xd, None, None, training=True, eps=1e-5)
    want.backward(dy.double())
    assert float((y - want.detach()).norm() / want.detach().norm()) <= 1e-6 and float((dx - xd.grad).norm() / xd.grad.norm()) <= 3e-6


def test_training_batch_norm_in_a_cluster_beyond_2_to_30_elements(capi):
    """Ragged planes of a tensor whose bytes do not fit 32 bits: the channel whose first elements are 2^30 elements from the tensor's end,
    those next to it and those at both ends, against float64 arithmetic (tolerances as above)."""
    n, c, h, w = 4, 368228, 27, 27
    total = n * c * h * w
    assert 2 ** 30 < total < 2 ** 31
    if torch.cuda.mem_get_info()[0] < 24 * 2 ** 30:
        pytest.skip("needs 24 GiB of device memory")
    g = torch.Generator(device="cuda")
    g.manual_seed(30)
    x, dy = (torch.empty((n, c, h, w), device="cuda").normal_(mu, 1.5, generator=g) for mu in (1.0, 0.0))
    gamma = torch.empty(c, device="cuda").uniform_(0.5, 1.5, generator=g)
    beta = torch.empty(c, device="cuda").normal_(0.0, 0.1, generator=g)
    y, dx = (torch.full_like(x, float("nan")) for _ in range(2))
    saved, sums, bsums = (torch.empty(k * c, device="cuda") for k in (2, 2, 3))
    ws = torch.empty(capi.bn_train_workspace_bytes(n, c, h * w), dtype=torch.uint8, device="cuda")
    capi.bn_train_fwd(y, saved, sums, x, gamma, beta, 1e-5, [], workspace=ws)
    capi.bn_train_bwd(dx, bsums, dy, x, gamma, beta, saved, [], workspace=ws)
    at = (total - 2 ** 30) // (h * w)
    pick = torch.tensor([0, 1, at - 1, at, at + 1, c - 2, c - 1], device="cuda")
    xd, ga, be = (t[:, pick].double().requires_grad_(True) if t is x else t[pick].double().requires_grad_(True) for t in (x, gamma, beta))
    want = torch.nn.functional.batch_norm(xd, None, None, ga, be, training=True, eps=1e-5)
    want.backward(dy[:, pick].double())
    norm = lambda t: (t * t).sum((0, 2, 3)).sqrt()
    assert bool((norm(y[:, pick].double() - want) <= 1e-6 * norm(want)).all())
    assert bool((norm(dx[:, pick].double() - xd.grad) <= 3e-6 * norm(xd.grad)).all())
    assert not bool(torch.isnan(y.view(-1)).any()) and not bool(torch.isnan(dx.view(-1)).any())


def test_host_threads_launch_clusters_of_different_sizes(capi):
    """Two threads, each on its own stream, with channels that need 50 KB and 512 bytes of shared memory per CTA (twice that backward) in the same
    instantiation: a launch does not depend on what the other thread's needs. Same results as from one thread."""
    import threading

    def state(shape, seed):
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        c = shape[1]
        x, dy = (torch.empty(shape, device="cuda").normal_(generator=g) for _ in range(2))
        gamma, beta = torch.ones(c, device="cuda"), torch.zeros(c, device="cuda")
        y, dx = torch.empty_like(x), torch.empty_like(x)
        saved, sums, bsums = (torch.empty(k * c, device="cuda") for k in (2, 2, 3))
        ws = torch.empty(capi.bn_train_workspace_bytes(shape[0], c, shape[2] * shape[3]), dtype=torch.uint8, device="cuda")
        return x, dy, gamma, beta, y, dx, saved, sums, bsums, ws, torch.cuda.Stream()

    def step(s):
        x, dy, gamma, beta, y, dx, saved, sums, bsums, ws, stream = s
        capi.bn_train_fwd(y, saved, sums, x, gamma, beta, 1e-5, [], workspace=ws, stream=stream)
        capi.bn_train_bwd(dx, bsums, dy, x, gamma, beta, saved, [], workspace=ws, stream=stream)

    states = [state((16, 160, 28, 28), 1), state((2, 160, 8, 8), 2)]
    torch.cuda.synchronize()
    want = []
    for s in states:
        step(s)
        want.append([host(t).copy() for t in (s[4], s[5], s[6], s[8])])
    failures = []

    def work(s):
        try:
            for _ in range(4000):
                step(s)
        except Exception as e:
            failures.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in states]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failures, failures
    for s, w in zip(states, want):
        for t, a in zip((s[4], s[5], s[6], s[8]), w):
            assert_bits_equal(host(t), a, "threads")


def test_tanh_vectors_with_large_exponents(capi, oracle):
    """Vectors of which no, one or every element's exponent is beyond 2^126, up to overflow, infinities and NaN."""
    g = synth.rng(1, salt=77)
    x = synth.normal(g, (3, 4, 8, 8), 0.0, 20.0)
    x.reshape(-1)[::7] *= 40.0
    x[0, 0, 0] = [43.4, 43.6, 44.3, 44.4, 87.0, -87.0, 1e30, -1e30]
    x[0, 0, 1, :5] = [np.inf, -np.inf, np.nan, 0.0, -0.0]
    one, zero = np.ones(4, np.float32), np.zeros(4, np.float32)
    y = torch.empty(x.shape, device="cuda")
    capi.bn_infer_act(y, dev(x), bn=[dev(a) for a in (one, zero, zero, one)], acts=[capi.tanh(1.0, 1.0)])
    want = oracle.tanh_fwd(x, 1.0, 1.0)
    got = host(y)
    assert (np.isnan(got) == np.isnan(want)).all()
    ok = ~np.isnan(want)
    # the exponential is good to 2^-22 + 6e-8 |2 x| relative, which a quotient near 1 hardly sees
    assert np.abs(got[ok] - want[ok]).max() <= 1e-6


def test_training_batch_norm_replayed_from_a_graph(capi, tuning):
    """The launch of statistics, finishing and apply items, captured once and replayed with other inputs in the same buffers: nothing
    that an earlier replay left in the workspace may pass for this one's."""
    tuning("chain_cluster", 99)
    shape = (64, 24, 28, 28)
    c = shape[1]
    x, dy, y, dx = (torch.zeros(shape, device="cuda") for _ in range(4))
    gamma, beta = torch.full((c,), 1.25, device="cuda"), torch.full((c,), 0.1, device="cuda")
    saved, sums, bsums = (torch.zeros(k * c, device="cuda") for k in (2, 2, 3))
    ws = torch.zeros(capi.bn_train_workspace_bytes(shape[0], c, 784), dtype=torch.uint8, device="cuda")

    def step():
        capi.bn_train_fwd(y, saved, sums, x, gamma, beta, 1e-5, [capi.relu()], workspace=ws)
        capi.bn_train_bwd(dx, bsums, dy, x, gamma, beta, saved, [capi.relu()], workspace=ws)

    step()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        step()
    for k in range(4):
        x.normal_(float(k), 1.0 + k)
        dy.normal_()
        graph.replay()
        got = [host(t).copy() for t in (y, saved, dx, bsums)]
        step()
        for a, t in zip(got, (y, saved, dx, bsums)):
            assert_bits_equal(a, host(t), "replay %d" % k)
