"""Properties of kernel sources that no run on a sound machine shows."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zoph_rnn_b200", "csrc")


def body(name, start, end):
    with open(os.path.join(CSRC, name)) as f:
        s = re.sub(r"//[^\n]*", "", f.read())
    i = s.index(start)
    return s[i:s.index(end, i)]


def test_a_split_link_that_gave_up_waits_for_its_partner():
    """The halves of a split tile travel with asynchronous stores into another CTA's shared memory.  A CTA that ends in order has waited for
    them; one whose wait gave up must not leave before the others' threads have ended or arrived: a cluster barrier at the end of the
    kernel, by all threads, on the flag that every wait sets when it gives up."""
    s = body("tc_link.cu", "void link_body(", "template <int BN, int MODE, int EPI, int SPLIT>\n__global__")
    end = s[s.index("tcgen05.dealloc"):]
    steps = [end.index(t) for t in ("if (SPLIT > 1 && ct.abort) {", "cluster_arrive();", "cluster_wait();", "settle_copies();")]
    assert steps == sorted(steps)
    # every bounded wait of the kernel reports through that flag, and no thread looks at it before all of them are over
    waits = re.findall(r"mbar_wait(?:_cluster)?\(([^;]*?), p\.err, \d\)", s)
    assert len(waits) == len(re.findall(r"\bmbar_wait(?:_cluster)?\(", s)) and all(w.endswith("&ct.abort") for w in waits)
    assert s.rindex("__syncthreads()") > s.rindex("mbar_wait")


def test_no_early_mask_can_name_the_fed_back_attention_output():
    """Bit s of a cell's early mask lets its kernel read source s before the launch ahead has ended.  Source 2, the fed-back attention output,
    is what that launch writes, so no flag that travels in such a mask may have its bit (nor a higher one: the mask's users count bits),
    and a mask that has one all the same is refused before anything is launched."""
    with open(os.path.join(CSRC, "zrnn_api.cu")) as f:
        s = re.sub(r"//[^\n]*", "", f.read())
    flags = {}
    for enum in re.findall(r"enum \{([^{}]*\bEARLY_X\b[^{}]*)\}", s):
        for name, value in re.findall(r"(\w+) = ([^,]+)", enum):
            flags[name] = eval(value, {}, flags)
    assert {"EARLY_X": 1, "EARLY_H": 2}.items() <= flags.items()
    assert all(v & ~3 == 0 for v in flags.values()), flags
    # every mask of a caller is made of these flags, and cell_forward looks at it before it does anything
    cell = body("zrnn_api.cu", "int cell_forward(", "\n}")
    assert re.search(r"\{\s*if \(early & ~EARLY_ANY\) return fail\(", cell)
    assert flags["EARLY_ANY"] == 3


def test_softmax_sums_use_full_precision_exponentials():
    """The sums of the vocabulary softmax are fp32 in every mode, whatever its operands are rounded to: expf, no faster function of a larger
    error.  (One unit of the last place of a sum of at least 1 hides the difference, so no output shows it.)"""
    for name in ("tc_vocab.cu", "tc_vocab_pair.cu", "tc_gemm.cu"):
        with open(os.path.join(CSRC, name)) as f:
            s = re.sub(r"//[^\n]*", "", f.read())
        assert "expf(" in s
        assert not re.search(r"__expf|__exp10f|exp2f|ex2\.approx|__powf|use_fast_math", s), name
    with open(os.path.join(os.path.dirname(CSRC), "build.py")) as f:
        assert "use_fast_math" not in f.read()


def test_launch_rules_ask_the_current_device_for_its_multiprocessors():
    """One function keeps the count, per device and safe for several threads; no rule has a count of its own or the first device's."""
    asks = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                s = re.sub(r"//[^\n]*", "", f.read())
            asks[name] = s.count("cudaDevAttrMultiProcessorCount")
            if name in ("tc_chain.cu", "tc_vocab.cu", "tc_vocab_pair.cu", "tc_cell_pair.cu"):
                assert not re.search(r"\b(147|148|73|74)\b", s), name
    assert {k: v for k, v in asks.items() if v} == {"tc_gemm.cu": 1}
    assert "std::atomic<int> count[kMaxDevices]" in body("tc_gemm.cu", "int device_sms()", "\n}")


def test_the_persistent_decoder_requests_the_weights_of_its_last_k_blocks():
    """Its activation ring may hold more k-blocks than its weight ring.  A producer that left with the last activation requested would, if the
    MMAs had not freed a weight stage by then, leave the last k-blocks without weights, and the kernel would wait for them until its bounded
    waits give up."""
    s = body("tc_decoder.cu", "if (warp == 8) {", "else if (warp == 9)")
    loop = s[s.index("while ("):]
    assert loop.startswith("while (!ac.end || !wc.end) {")
    weights, acts = loop.index("!wc.end && w_it < a_it + NW"), loop.index("if (!ac.end) {")
    assert weights < acts < loop.index("ac.pl")  # (and no activation is looked at beyond the last)


def test_gemm_packs_its_weights_before_the_launch_ahead_of_the_product():
    """A link kernel requests its weights before it waits for the launch ahead of it.  In the stand-alone product the weights are packed by a
    launch of the same call, so another launch, which waits for that one, has to lie between."""
    s = body("zrnn_api.cu", "int zrnn_gemm(", "zrnn_tc_error()")
    assert s.index("launch_pack_weights(") < s.index("launch_convert_rows(") < s.index("launch_tc_chain(")


def test_a_cta_with_all_of_the_tensor_memory_and_a_partner_has_its_sm_for_itself():
    """Two kernels of different streams whose CTAs wait for their cluster partners must not hold the tensor memory that the other one's
    partner waits for: a kernel that allocates all 512 columns and has partners asks for (nearly) all of an SM's shared memory.  That the
    constant is large enough is a static_assert beside it; here: that it is what these launches ask for, and that no other kernel with
    cluster partners allocates all columns."""
    for name, constant, when in (("tc_link.cu", "kWholeSm", r"WHOLE && SPLIT > 1 \? \(size_t\)kWholeSm :"), ("tc_vocab_pair.cu", "kSmem", None), ("tc_cell_pair.cu", "kSmem", None)):
        with open(os.path.join(CSRC, name)) as f:
            whole = re.sub(r"\s+", " ", re.sub(r"//[^\n]*", "", f.read()))
        assert "static_assert(fills_sm(%s)," % constant in whole
        launch = re.sub(r"\s+", " ", body(name, "cudaError_t launch_t(", "cudaLaunchKernelEx"))
        asked = re.search(r"cfg\.dynamicSmemBytes = (\w+);", launch).group(1)
        if when:
            assert re.search(r"const size_t %s = %s" % (asked, when), launch)
        else:
            assert asked == constant
    with_partners = {n for n in os.listdir(CSRC) if n.endswith(".cu") and "tcgen05.alloc" in open(os.path.join(CSRC, n)).read() + "\n"
                     and re.search(r"__cluster_dims__|ClusterDimension", open(os.path.join(CSRC, n)).read())}
    assert with_partners == {"tc_link.cu", "tc_decoder.cu"}  # (the pair kernels allocate through tc_pair_device.cuh)
    assert "static_assert(fills_sm(dec_smem(TC_BF16))" in open(os.path.join(CSRC, "tc_decoder.cu")).read()
