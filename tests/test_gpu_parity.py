"""GPU parity tests: the CUDA path, called through the C ABI, against the golden
fixtures (made from the unmodified reference definition) and against the oracle
on the same seeded inputs.

Bars:
* expert selection (as sets), histogram, offsets and the permutation: bit-exact;
* combination weights: relative 1e-6 (fp32 summation order of eight terms);
* bf16 output: cosine >= 0.9999 and max-abs error <= 2e-2 x output RMS.  The
  definition's own fp32 summation-order noise (~1e-5 relative) already flips the
  final bf16 rounding of about 0.5 % of the elements, and ONE bf16 step of an
  element with |x| >= 1 is 0.0078 or more, i.e. above 2e-2 x RMS for these
  workloads.  The max-abs bar is therefore applied literally to every element
  except those that differ from the reference by exactly one bf16 step, and those
  must satisfy the tighter fp32-domain bar |out - ref_fp32| <= half a bf16 step
  + 2e-3 x RMS (the result is a correct rounding of a value within a tenth of the
  tolerance of the reference's pre-cast fp32 value).  Both numbers are printed.
"""
import json
import os

import numpy as np
import pytest
import torch

import moe_oracle
import ws_readers

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
TOL_MAX_ABS_OVER_RMS = 2e-2
TOL_COSINE = 0.9999
TOL_F32_DOMAIN_OVER_RMS = 2e-3
RSF = 2.5


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    torch.backends.cuda.matmul.allow_tf32 = False
    return torch.device("cuda", 0)


@pytest.fixture(scope="module")
def W(pkg, dev):
    return pkg.gen.make_shard_weights(0, dev)


def run_op(pkg, tok, W, offset, rsf=RSF, out=None):
    out = pkg.op.run(tok.routing_logits, tok.routing_bias, tok.hidden_states, tok.hidden_states_scale,
                     W.gemm1_weights, W.gemm1_weights_scale, W.gemm2_weights, W.gemm2_weights_scale, offset, rsf, out)
    assert pkg.op.kernel_status() == 0, "a kernel recorded an error bit"
    return out


def bf16_step(x: torch.Tensor) -> torch.Tensor:
    ax = x.abs().double().clamp_min(2.0 ** -126)
    return torch.pow(2.0, torch.floor(torch.log2(ax)) - 7)


def assert_output_close(out_bf16, ref_bf16, ref_f32, rms=None):
    """The bars of the module docstring; arithmetic on the device of ``out_bf16`` in row chunks."""
    dev = out_bf16.device
    ref_bf16, ref_f32 = ref_bf16.to(dev), ref_f32.to(dev)
    m = moe_oracle.output_metrics(out_bf16, ref_bf16, ref_f32)
    if rms is None:
        rms = float(torch.sqrt((ref_f32.double() ** 2).mean())) if ref_f32.numel() else 0.0
    print("parity:", json.dumps(moe_oracle.parity_report(m)))
    assert m["cosine"] >= TOL_COSINE
    if rms == 0.0:
        assert float(out_bf16.float().abs().max()) == 0.0
        return m
    steps = moe_oracle.bf16_steps(out_bf16, ref_bf16)
    rows = max(1, (1 << 23) // out_bf16.shape[-1])
    for r0 in range(0, out_bf16.shape[0], rows):
        out = out_bf16[r0:r0 + rows].double()
        err = (out - ref_bf16[r0:r0 + rows].double()).abs()
        literal_bad = err > TOL_MAX_ABS_OVER_RMS * rms
        one_step = steps[r0:r0 + rows] == 1
        assert bool((~literal_bad | one_step).all()), \
            f"{int((literal_bad & ~one_step).sum())} elements beyond 2e-2 x RMS that are not single rounding flips"
        f32_err = (out - ref_f32[r0:r0 + rows].double()).abs()
        bound = 0.5 * bf16_step(out) + TOL_F32_DOMAIN_OVER_RMS * rms
        assert bool((f32_err <= bound).all()), f"fp32-domain error {float((f32_err - bound).max())} over the bound"
    return m


def assert_selection_and_permutation(pkg, T, ref_topk_sorted, ref_counts, ref_offsets, ref_perm_token, ref_perm_weight):
    im = ws_readers.intermediates(pkg, T, stages=T <= 1024)
    got = torch.sort(im["topk_idx"].long(), dim=1).values
    assert torch.equal(got, torch.as_tensor(ref_topk_sorted).long()), "expert selection differs"
    assert torch.equal(im["counts"].long(), torch.as_tensor(ref_counts).long())
    assert torch.equal(im["offs"].long(), torch.as_tensor(ref_offsets).long())
    assert torch.equal(im["perm_token"].long(), torch.as_tensor(ref_perm_token).long()), "permutation differs"
    torch.testing.assert_close(im["perm_weight"], torch.as_tensor(ref_perm_weight), rtol=1e-6, atol=1e-9)
    return im


@pytest.mark.parametrize("name", ["cpu_ref_t8", "decode_t1", "skew_t64", "offset64_t8", "ragged_t37", "prefill_t4096"])
def test_golden_fixture(pkg, dev, W, name):
    z = np.load(os.path.join(GOLDEN, name + ".npz"))
    meta = json.loads(str(z["meta"]))
    T = meta["T"]
    tok = pkg.gen.make_tokens(T, meta["token_seed"], dev, meta["skew"])
    # the generator is device independent: same bytes as the fixture's CPU inputs
    assert pkg.gen.digest(tok.routing_logits, tok.routing_bias, tok.hidden_states,
                          tok.hidden_states_scale) == meta["tokens_digest"]
    for le in (0, 5, 31):
        assert pkg.gen.digest(W.gemm1_weights[le], W.gemm1_weights_scale[le], W.gemm2_weights[le],
                              W.gemm2_weights_scale[le]) == meta["weights_digest"][f"w_expert{le}"]
    out = run_op(pkg, tok, W, meta["local_expert_offset"], meta["routed_scaling_factor"])
    assert_selection_and_permutation(pkg, T, z["topk_sorted"].astype(np.int64), z["counts"], z["offsets"],
                                     z["perm_token"], z["perm_weight"])
    rows = torch.as_tensor(z["rows"]).long()
    ref_bf16 = torch.as_tensor(z["out_bf16"].view(np.int16)).view(torch.bfloat16)
    assert_output_close(out[rows.to(dev)], ref_bf16, torch.as_tensor(z["out_f32"]), rms=meta["out_rms"])


LIVE_CASES = [
    # T, token seed, skew, local_expert_offset
    (1, 0, False, 0),        # no local expert at all: all-zero output
    (2, 5, False, 32),
    (3, 7, False, 224),      # last shard
    (5, 11, True, 0),        # decode kernel, several tokens per expert
    (9, 14, False, 128),
    (13, 12, False, 0),      # more tokens than routing warps in the decode kernel
    (16, 1, False, 0),
    (16, 13, True, 0),       # decode kernel at its largest: 128 rows on 8 experts
    (17, 2, False, 96),
    (33, 4, True, 0),        # every token lands on 8 local experts
    (127, 6, False, 0),
    (128, 6, False, 160),
    (129, 6, True, 0),       # > 64 tokens per expert: two 64-wide... and 128-wide token tiles
    (300, 0, True, 0),       # 150 tokens per expert: crosses a 128-token tile
    (512, 8, False, 64),
    (1000, 9, False, 0),
]


@pytest.mark.parametrize("T,seed,skew,offset", LIVE_CASES)
def test_against_oracle(pkg, dev, W, T, seed, skew, offset):
    tok = pkg.gen.make_tokens(T, seed, dev, skew)
    out = run_op(pkg, tok, W, offset)
    ref = moe_oracle.run_full(tok.routing_logits, tok.routing_bias, tok.hidden_states, tok.hidden_states_scale,
                              W.gemm1_weights, W.gemm1_weights_scale, W.gemm2_weights, W.gemm2_weights_scale,
                              offset, RSF)
    im = assert_selection_and_permutation(pkg, T, torch.sort(ref.topk_idx.cpu(), dim=1).values, ref.counts,
                                          ref.offsets, ref.perm_token, ref.perm_weight.cpu())
    assert im["n_sel"] == int(ref.counts.sum())
    assert_output_close(out, ref.output, ref.output_f32)
    # tokens with no local expert are exact zeros (the output needs no memset by the caller)
    no_local = torch.as_tensor(im["local_mask"] == 0)
    assert float(out[no_local.to(dev)].float().abs().max() if bool(no_local.any()) else 0.0) == 0.0


@pytest.mark.parametrize("T", [16, 200, 1024, 1100, 2048])
def test_every_token_on_the_same_eight_local_experts(pkg, dev, W, T):
    """The case the workspace is sized for: a bias that makes every token select local experts 0..7, so the call has
    8 T rows (the row capacity) on eight experts with T rows each: the largest tiles-per-expert count of every path."""
    tok = pkg.gen.make_tokens(T, 31, dev)
    bias = tok.routing_bias.float()
    bias[:8] += 10.0
    tok.routing_bias = bias.to(torch.bfloat16)
    out = run_op(pkg, tok, W, 0)
    ref = moe_oracle.run_full(tok.routing_logits, tok.routing_bias, tok.hidden_states, tok.hidden_states_scale,
                              W.gemm1_weights, W.gemm1_weights_scale, W.gemm2_weights, W.gemm2_weights_scale, 0, RSF)
    assert ref.counts[:8].tolist() == [T] * 8 and int(ref.counts.sum()) == 8 * T
    im = assert_selection_and_permutation(pkg, T, torch.sort(ref.topk_idx.cpu(), dim=1).values, ref.counts,
                                          ref.offsets, ref.perm_token, ref.perm_weight.cpu())
    assert im["n_sel"] == 8 * T
    assert_output_close(out, ref.output, ref.output_f32)


@pytest.mark.parametrize("T,seed,offset", [(8192, 21, 0), (16384, 0, 0)])
def test_large_batch_against_gpu_oracle(pkg, dev, W, T, seed, offset):
    """Shard calls of the size one rank of the expert-parallel layer sees (8-24 k rows): 128-token tiles,
    the multi-CTA permutation fill.  The oracle runs on the GPU in fp32 (TF32 off): same definition,
    cuBLAS fp32 summation order instead of the CPU's."""
    tok = pkg.gen.make_tokens(T, seed, dev)
    out = run_op(pkg, tok, W, offset)
    ref = moe_oracle.run_full(tok.routing_logits, tok.routing_bias, tok.hidden_states, tok.hidden_states_scale,
                              W.gemm1_weights, W.gemm1_weights_scale, W.gemm2_weights, W.gemm2_weights_scale,
                              offset, RSF)
    im = assert_selection_and_permutation(pkg, T, torch.sort(ref.topk_idx.cpu(), dim=1).values, ref.counts,
                                          ref.offsets, ref.perm_token, ref.perm_weight.cpu())
    assert im["n_sel"] == int(ref.counts.sum()) and im["n_sel"] > 4000
    assert_output_close(out, ref.output, ref.output_f32)


def test_definition_on_gpu_against_definition_on_cpu(pkg, dev):
    """How far apart are two faithful fp32 evaluations of the definition?  The oracle on the GPU (cuBLAS fp32,
    TF32 off) against the oracle on the CPU, T = 64, skewed routing (512 rows).  Neither is the CUDA path; the
    printed numbers show what the literal max-abs bar means for ANY implementation that does not share the
    reference's fp32 summation order, and are the yardstick for the flip census of the other tests."""
    T = 64
    tok = pkg.gen.make_tokens(T, 0, dev, True)
    active = list(range(16))
    Wg = pkg.gen.make_shard_weights(0, dev, experts=active)
    g = moe_oracle.run_full(tok.routing_logits, tok.routing_bias, tok.hidden_states, tok.hidden_states_scale,
                            Wg.gemm1_weights, Wg.gemm1_weights_scale, Wg.gemm2_weights, Wg.gemm2_weights_scale, 0, RSF)
    assert sorted(int(e) for e in g.counts.nonzero().squeeze(1)) == active
    cpu = lambda t: t.cpu()
    c = moe_oracle.run(cpu(tok.routing_logits), cpu(tok.routing_bias), cpu(tok.hidden_states),
                       cpu(tok.hidden_states_scale),
                       lambda le: tuple(cpu(x[le]) for x in (Wg.gemm1_weights, Wg.gemm1_weights_scale,
                                                              Wg.gemm2_weights, Wg.gemm2_weights_scale)), 0, RSF)
    m = moe_oracle.output_metrics(g.output, c.output, c.output_f32)
    print("oracle_gpu_vs_oracle_cpu:", json.dumps(moe_oracle.parity_report(m)))
    assert m["cosine"] >= TOL_COSINE and m["match_ratio"] == 1.0


@pytest.fixture
def options(pkg):
    """Sets the operator's process-wide options for one test and restores the default afterwards."""
    yield pkg.loader.set_options
    pkg.loader.set_options(0)


@pytest.mark.parametrize("T,seed,skew", [(4096, 0, False), (1500, 2, True)])
def test_fused_large_batch_path_against_unfused_path(pkg, dev, W, options, T, seed, skew):
    """More than 1024 tokens: GEMM1 with SwiGLU and the plane split in its epilogue against the multi-kernel path
    (GEMM1 -> SwiGLU kernel) on the same inputs.  Both apply the same fp32 operations in the same order to every
    element, so the e4m3 planes and their scales must agree bit for bit; the outputs (deterministic combine in
    both) may differ by the tensor core's internal summation order only."""
    tok = pkg.gen.make_tokens(T, seed, dev, skew)
    options(pkg.loader.OPT_UNFUSED)
    out_u = run_op(pkg, tok, W, 0).clone()
    cq_u, cs_u = ws_readers.swiglu_planes(pkg, T)
    options(0)
    out_f = run_op(pkg, tok, W, 0).clone()
    cq_f, cs_f = ws_readers.swiglu_planes(pkg, T)
    assert cq_u.shape[1] > 1024
    assert torch.equal(cs_u, cs_f), "plane scales differ"
    assert torch.equal(cq_u, cq_f), f"{int((cq_u != cq_f).sum())} plane bytes differ"
    steps = moe_oracle.bf16_steps(out_f, out_u)
    print("fused_vs_unfused_output:", json.dumps({"n_diff": int((steps > 0).sum()), "max_steps": int(steps.max())}))
    m = moe_oracle.output_metrics(out_f, out_u, out_u.float())
    assert m["cosine"] >= 0.999999 and m["match_ratio"] == 1.0


def check_rows_per_expert(pkg, dev, W, T, counts):
    """A batch of T tokens in which expert e of the shard gets exactly `counts[e]` rows and no other expert any: the first
    sum(counts) tokens select one local expert each, the others none.  Same bars as every other batch against the
    oracle; that the batch is what it is meant to be is checked on the oracle's and on the operator's side."""
    tok = pkg.gen.make_tokens(T, 11, dev)
    logits = tok.routing_logits * 0.01 - 6.0
    logits[:, 32:35] += 12.0                      # seven experts of groups 1 to 3 for everybody
    logits[:, 64:66] += 12.0
    logits[:, 96:98] += 12.0
    logits[:, 130] += 6.0                         # the eighth, where no local expert scores higher
    expert = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts)).to(dev)
    logits[torch.arange(len(expert), device=dev), expert] += 12.0
    bias = torch.zeros_like(tok.routing_bias)
    ref = moe_oracle.run_full(logits, bias, tok.hidden_states, tok.hidden_states_scale, W.gemm1_weights,
                              W.gemm1_weights_scale, W.gemm2_weights, W.gemm2_weights_scale, 0, RSF)
    want = counts + [0] * (32 - len(counts))
    assert ref.counts.tolist() == want
    out = pkg.op.run(logits, bias, tok.hidden_states, tok.hidden_states_scale, W.gemm1_weights, W.gemm1_weights_scale,
                     W.gemm2_weights, W.gemm2_weights_scale, 0, RSF)
    assert pkg.op.kernel_status() == 0
    assert list(pkg.op.read_schedule(T).counts) == want
    assert_output_close(out, ref.output, ref.output_f32)
    assert float(out[sum(counts):].float().abs().max()) == 0.0


@pytest.mark.parametrize("fast_combine", [False, True])
@pytest.mark.parametrize("counts", [[1, 31, 32, 33, 64, 65, 96, 97, 127, 128, 129, 160], [255, 256, 257, 1]])
def test_ragged_token_tiles_of_the_large_batch_path(pkg, dev, W, options, counts, fast_combine):
    """Experts whose row counts sit at the edges of the 32-row steps and of the 128-token tiles, with both combines."""
    options(pkg.loader.OPT_FAST_COMBINE if fast_combine else 0)
    check_rows_per_expert(pkg, dev, W, max(1100, sum(counts) + 5), counts)


@pytest.mark.parametrize("T,counts", [
    (30, [1, 15]), (30, [16, 2, 8]), (32, [17, 14]),                   # 32-token tiles in both GEMMs, one launch routes
    (64, [1, 15, 16, 17]), (64, [31, 32]), (60, [48, 7]), (64, [49, 1]),   # GEMM1 on 64-token tiles, GEMM2 on 32
    (200, [1, 15, 16, 17, 31, 32, 33]), (200, [47, 48, 49]),          # 32 / 32 with several tiles an expert
    (700, [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 113]),  # 64 / 32
    (900, [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 127, 128, 129]),   # 64 / 64
])
def test_ragged_token_tiles_up_to_1024_tokens(pkg, dev, W, T, counts):
    """Experts whose row counts sit at the edges of the 16-row steps and of the 32- and 64-token tiles of the multi-kernel
    path, where the number of rows an item brings sets the distance of GEMM2's planes in TMEM, which scales are copied
    and which promotion warps read nothing."""
    check_rows_per_expert(pkg, dev, W, T, counts)


@pytest.mark.parametrize("T,seed,skew,offset", [(4096, 0, False, 0), (1100, 3, True, 0), (6000, 5, False, 96)])
def test_fast_combine_against_oracle(pkg, dev, W, options, T, seed, skew, offset):
    """MOE_B200_OPT_FAST_COMBINE: routing-weight multiply and fp32 combine in GEMM2's epilogue (vector reductions,
    last-arriver bf16 cast).  Same bars as the deterministic path against the oracle; rows of tokens without a
    local expert are exact zeros; twice in a row on the same workspace (the accumulator is cleared per call)."""
    tok = pkg.gen.make_tokens(T, seed, dev, skew)
    ref = moe_oracle.run_full(tok.routing_logits, tok.routing_bias, tok.hidden_states, tok.hidden_states_scale,
                              W.gemm1_weights, W.gemm1_weights_scale, W.gemm2_weights, W.gemm2_weights_scale,
                              offset, RSF)
    options(pkg.loader.OPT_FAST_COMBINE)
    for _ in range(2):
        out = torch.full((T, 7168), 7.0, dtype=torch.bfloat16, device=dev)
        run_op(pkg, tok, W, offset, out=out)
        assert_output_close(out, ref.output, ref.output_f32)
        _, _, mask = pkg.op.route(tok.routing_logits, tok.routing_bias, offset, RSF)
        no_local = mask == 0
        assert (T == 1100 or bool(no_local.any())) and float(out[no_local].float().abs().max() if bool(no_local.any()) else 0.0) == 0.0
    options(0)
    det = run_op(pkg, tok, W, offset).clone()
    steps = moe_oracle.bf16_steps(out, det)
    print("fast_vs_deterministic:", json.dumps({"n_diff": int((steps > 0).sum()), "n": out.numel()}))
    assert int((steps > 0).sum()) < 0.02 * out.numel()


def test_empty_batch_is_a_noop(pkg, dev, W):
    tok = pkg.gen.make_tokens(0, 0, dev)
    out = pkg.op.run(tok.routing_logits, tok.routing_bias, tok.hidden_states, tok.hidden_states_scale,
                     W.gemm1_weights, W.gemm1_weights_scale, W.gemm2_weights, W.gemm2_weights_scale, 0, RSF)
    assert out.shape == (0, 7168)


def test_full_size_properties(pkg, dev, W):
    """Size-independent properties at the prefill size (T = 4096):
    run-to-run determinism, exact power-of-two linearity in the scaling factor,
    and equivariance under a permutation of the tokens."""
    T = 4096
    tok = pkg.gen.make_tokens(T, 0, dev)
    a = run_op(pkg, tok, W, 0).clone()
    b = run_op(pkg, tok, W, 0).clone()
    assert torch.equal(a.view(torch.int16), b.view(torch.int16)), "two runs differ: the combine is not deterministic"
    c = run_op(pkg, tok, W, 0, rsf=2 * RSF).clone()
    assert torch.equal((a.float() * 2).to(torch.bfloat16).view(torch.int16), c.view(torch.int16))
    perm = torch.randperm(T, generator=torch.Generator().manual_seed(1)).to(dev)
    tok_p = type(tok)(tok.routing_logits[perm].contiguous(), tok.routing_bias, tok.hidden_states[perm].contiguous(),
                      tok.hidden_states_scale[:, perm].contiguous())
    d = run_op(pkg, tok_p, W, 0)
    assert torch.equal(d.view(torch.int16), a[perm].view(torch.int16)), "output depends on the position of a token"


def test_host_buffer_entry_point(pkg, dev, W):
    """moe_fp8_block_scale_run_host: pinned host token tensors in, host output out."""
    T = 8
    tok = pkg.gen.make_tokens(T, 0, dev)
    want = run_op(pkg, tok, W, 0).cpu()
    pin = lambda t: t.cpu().pin_memory()
    out_h = torch.empty(T, 7168, dtype=torch.bfloat16).pin_memory()
    pkg.op.run_host(pin(tok.routing_logits), pin(tok.routing_bias), pin(tok.hidden_states),
                    pin(tok.hidden_states_scale), W.gemm1_weights, W.gemm1_weights_scale, W.gemm2_weights,
                    W.gemm2_weights_scale, 0, RSF, out_h)
    assert torch.equal(out_h.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("T", [1, 8, 64, 1100])
def test_cuda_graph_replay(pkg, dev, W, T):
    """The operator call recorded in a CUDA graph (after one ordinary call) and replayed over new values in the
    same buffers gives the bits of ordinary calls, replay after replay: all launch state that changes from call
    to call lives on the device (the decode kernel's barrier tag among it)."""
    gen = pkg.gen
    toks = [gen.make_tokens(T, seed, dev) for seed in (11, 12, 13)]
    want = [run_op(pkg, t, W, 0).clone() for t in toks]
    buf = gen.make_tokens(T, 11, dev)
    out = torch.empty(T, 7168, dtype=torch.bfloat16, device=dev)
    run_op(pkg, buf, W, 0, out=out)                      # sizes the workspace, fills the tensor-map cache
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pkg.op.run(buf.routing_logits, buf.routing_bias, buf.hidden_states, buf.hidden_states_scale,
                   W.gemm1_weights, W.gemm1_weights_scale, W.gemm2_weights, W.gemm2_weights_scale, 0, RSF, out)
    for rep in range(2):
        for t, w in zip(toks, want):
            buf.routing_logits.copy_(t.routing_logits)
            buf.routing_bias.copy_(t.routing_bias)
            buf.hidden_states.view(torch.uint8).copy_(t.hidden_states.view(torch.uint8))
            buf.hidden_states_scale.copy_(t.hidden_states_scale)
            out.zero_()
            graph.replay()
            graph.replay()                               # back to back: the second replay meets the first one's barrier word
            torch.cuda.synchronize()
            assert pkg.op.kernel_status() == 0
            assert torch.equal(out.view(torch.int16), w.view(torch.int16)), (T, rep)


def test_two_streams_with_their_own_workspaces(pkg, dev, W):
    """Calls on two streams, each with its own workspace, interleaved without waiting for one another: the library
    keeps no per-call state outside the workspace (its tensor-map cache is read-mostly and locked), so each stream
    gets the bits of a call made alone.  (Batches above 16 tokens: the decode kernel wants the device to itself.)"""
    op, gen = pkg.op, pkg.gen
    cases = [(300, 3), (1100, 4), (64, 5), (40, 6)]
    toks = [gen.make_tokens(T, seed, dev) for T, seed in cases]
    want = [run_op(pkg, t, W, 0).clone() for t in toks]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(device=dev) for _ in range(2)]
    spaces = [op.Workspace(dev) for _ in range(2)]
    outs = [torch.zeros_like(w) for w in want]
    for rep in range(3):
        for i, t in enumerate(toks):
            k = i % 2
            with torch.cuda.stream(streams[k]):
                op.run(t.routing_logits, t.routing_bias, t.hidden_states, t.hidden_states_scale, W.gemm1_weights,
                       W.gemm1_weights_scale, W.gemm2_weights, W.gemm2_weights_scale, 0, RSF, outs[i], workspace=spaces[k])
    torch.cuda.synchronize()
    for k in range(2):
        assert op.kernel_status(workspace=spaces[k]) == 0
    for o, w in zip(outs, want):
        assert torch.equal(o.view(torch.int16), w.view(torch.int16))


def test_workspace_too_small_is_reported(pkg, dev, W):
    tok = pkg.gen.make_tokens(8, 0, dev)
    out = torch.empty(8, 7168, dtype=torch.bfloat16, device=dev)
    ws = torch.empty(4096, dtype=torch.uint8, device=dev)
    rc = pkg.loader.lib.moe_fp8_block_scale_run(
        tok.routing_logits.data_ptr(), tok.routing_bias.data_ptr(), tok.hidden_states.data_ptr(),
        tok.hidden_states_scale.data_ptr(), W.gemm1_weights.data_ptr(), W.gemm1_weights_scale.data_ptr(),
        W.gemm2_weights.data_ptr(), W.gemm2_weights_scale.data_ptr(), 8, 0, RSF, out.data_ptr(),
        (ws.data_ptr() + 1023) // 1024 * 1024, 1024, None)
    assert rc == pkg.loader.EWORKSPACE


def test_fp8_umma_accumulation_known_answer(pkg, dev, W):
    """Known-answer check of the tensor-core path: with all-ones activations (scale 1) the
    GEMM1 result is the per-row sum of the dequantised weights, which fp64 gives exactly
    enough to expose a truncating or reduced-precision accumulator."""
    T = 16
    hs = torch.ones(T, 7168, device=dev).to(torch.float8_e4m3fn)
    hscale = torch.ones(56, T, device=dev)
    logits = torch.zeros(T, 256, device=dev)
    logits[:, 3] = 8.0          # every token picks local expert 3 first
    bias = torch.zeros(256, dtype=torch.bfloat16, device=dev)
    pkg.op.run(logits, bias, hs, hscale, W.gemm1_weights, W.gemm1_weights_scale, W.gemm2_weights,
               W.gemm2_weights_scale, 0, RSF)
    assert pkg.op.kernel_status() == 0
    im = ws_readers.intermediates(pkg, T)
    assert int(im["counts"][3]) == T
    rows = slice(int(im["offs"][3]), int(im["offs"][4]))
    w = W.gemm1_weights[3].double().view(32, 128, 56, 128) * W.gemm1_weights_scale[3].double()[:, None, :, None]
    want = w.sum(dim=(2, 3)).view(4096).cpu()
    got = im["g1"][rows].double()
    scale = float(w.abs().sum(dim=(2, 3)).max())
    assert float((got - want[None, :]).abs().max()) <= 2e-6 * scale


def test_tvm_ffi_entry_point_matches_c_abi(pkg, dev, W):
    """The harness-facing export `run` (tvm-ffi, the reference's binding) gives the same bits as the C ABI."""
    tvm_ffi = pytest.importorskip("tvm_ffi")
    lib = pkg.build.build_tvmffi()
    if lib is None:
        pytest.skip("tvm-ffi shim not built")
    mod = tvm_ffi.load_module(lib)
    for T, seed in ((8, 0), (130, 4)):
        tok = pkg.gen.make_tokens(T, seed, dev)
        want = run_op(pkg, tok, W, 32).clone()
        out = torch.zeros(T, 7168, dtype=torch.bfloat16, device=dev)
        mod.run(tok.routing_logits, tok.routing_bias, tok.hidden_states, tok.hidden_states_scale,
                W.gemm1_weights, W.gemm1_weights_scale, W.gemm2_weights, W.gemm2_weights_scale, 32, RSF, out)
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("T", [1, 7, 130, 4096])
def test_activation_quantisation_is_bit_exact(pkg, dev, T):
    """The quantisation kernel (the step before the operator) reproduces the generator's
    reference quantisation bit for bit: e4m3 bytes and the transposed [56, T] scales."""
    x = (pkg.gen.normal(21, 9, 0, T * 7168, dev).view(T, 7168) * 3.0).to(torch.bfloat16)
    x[0, :128] = 0                     # an all-zero block: scale floor, zeros out
    if T > 1:
        x[1, 5] = 30000.0              # a large outlier in a block
    q, s = pkg.op.quantize_activations(x.contiguous())
    q_ref, s_ref = pkg.gen.quant_1x128(x.to(torch.float32))
    assert torch.equal(s, s_ref.t().contiguous())
    assert torch.equal(q.view(torch.uint8), q_ref.view(torch.uint8))


def test_routing_randomised_against_oracle(pkg, dev):
    """Routing alone (moe_fp8_block_scale_route) on many random batches, bias scales and shard
    offsets: selected expert sets and the local-expert mask bit for bit, weights to 1e-6.
    Includes biases large enough to pin whole groups and logits with a narrow spread
    (many near-equal scores)."""
    g = torch.Generator().manual_seed(1234)
    total = 0
    for case in range(24):
        T = int(torch.randint(1, 700, (1,), generator=g))
        seed = int(torch.randint(0, 10 ** 6, (1,), generator=g))
        offset = 32 * int(torch.randint(0, 8, (1,), generator=g))
        tok = pkg.gen.make_tokens(T, seed, dev, skew=(case % 5 == 0))
        logits = tok.routing_logits * (0.05 if case % 3 == 0 else 1.0 if case % 3 == 1 else 4.0)
        bias = (tok.routing_bias.float() * (1.0 if case % 2 == 0 else 8.0)).to(torch.bfloat16)
        idx, w, mask = pkg.op.route(logits.contiguous(), bias, offset, RSF)
        ref_idx, ref_w = moe_oracle.routing(logits, bias, RSF)
        same = moe_oracle.selection_sets_equal(idx, ref_idx)
        if not bool(same.all()):
            gap_g, gap_e = moe_oracle.selection_margins(logits, bias)
            bad = (~same).nonzero().squeeze(1)
            # a mismatch is acceptable only on an exact tie, which torch.topk may break either way
            assert bool(((gap_g[bad.to(dev)] == 0) | (gap_e[bad.to(dev)] == 0)).all()), \
                f"selection differs on tokens {bad.tolist()} without a tie"
        ok = same.to(dev)
        torch.testing.assert_close(w[ok], ref_w.gather(1, idx.long())[ok], rtol=1e-6, atol=1e-9)
        local = ((ref_idx >= offset) & (ref_idx < offset + 32))
        want_mask = torch.where(local, torch.ones_like(ref_idx) << (ref_idx - offset).clamp(0, 31),
                                torch.zeros_like(ref_idx)).sum(dim=1)
        assert torch.equal(mask.long()[ok] & 0xFFFFFFFF, want_mask[ok] & 0xFFFFFFFF)
        total += T
    assert total > 1000
