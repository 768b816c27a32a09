"""Rules of the kernel sources that no run can show to be kept: what breaks when one is broken depends on how the lanes of a
warp happen to be scheduled, or on which cache a load is served from."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dqmoe_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())  # without comments


def braces(text, start):
    """The block that opens at the first '{' from `start` on."""
    at = text.index("{", start)
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError("unbalanced braces")


def test_roles_of_a_whole_warp_wait_together():
    """A role that one elected thread plays may poll a barrier alone. In one that a whole warp plays, a lane that goes on
    alone can let the barrier pass twice before another lane polls again, which then waits for a parity that is gone."""
    for name, roles in (("gemm_sm100.cu", ["else if (warp == 2)", "setmaxnreg_inc"]), ("gemm_mx_sm100.cu", ["setmaxnreg_inc"])):
        text = source(name)
        for role in roles:
            at = text.index(role)
            if role == "setmaxnreg_inc":
                at = text.rindex("else {", 0, at)
            body = braces(text, at)
            assert "mbar_wait_warp(" in body, (name, role)
            assert not re.search(r"\bmbar_wait\(", body), (name, role)


def test_buffers_are_released_by_a_converged_warp():
    """One lane arrives for its warp, so the others must be known to have read the buffer and to have seen the phase."""
    text = source("gemm_sm100.cu")
    release = braces(text, text.index("auto release_tmem"))
    assert release.index("__syncwarp()") < release.index("mbar_arrive")
    assert not re.search(r"if \(lane == 0\)\s*release_tmem", text)
    mx = source("gemm_mx_sm100.cu")
    for m in re.finditer(r"mbar_arrive\(&st\.(tmem_empty|overlap_free)", mx):
        assert "__syncwarp()" in mx[max(0, m.start() - 200):m.start()], mx[m.start() - 200:m.end()]


def test_dependents_read_their_predecessors_output_with_plain_loads():
    """A programmatic dependent is resident while the kernels before it still write what it reads behind its wait. Non-coherent
    loads (and what the compiler makes of const __restrict__ arguments) are for data that stays unchanged in that time."""
    found = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = source(name)
        for m in re.finditer(r"__global__", text):
            signature = text[m.start():text.find("{", m.start())]
            if ";" in signature:
                continue
            body = braces(text, m.start())
            if not re.search(r"\b(pdl_enter|pdl_wait|wait_for_primary)\(", body):
                continue
            found += 1
            for word in ("__restrict__", "__ldg", "ld_nc16", ".nc"):
                assert word not in signature + body, (name, signature[:120], word)
        if name in ("permute.cu", "quant.cu", "quant_mx.cu"):  # device helpers of such kernels
            assert "ld_nc16" not in text and "__ldg" not in text, name
    assert found >= 18


def test_block_scales_are_passed_on_by_a_release():
    """Block mode's scales arrive on the stage's barrier, which only the MMA thread observes; the epilogue warps read them behind
    the accumulator buffer's. A tcgen05.commit tracks the completion of MMAs and publishes nothing else, so the thread arrives
    there itself, and on the barrier that lets the ring slot be refilled."""
    text = source("gemm_sm100.cu")
    at = text.index("else if (warp == 1)", text.index("setmaxnreg_dec"))
    issuer = braces(text, at)
    block = issuer[issuer.index("acc_it) {", issuer.index("} else {\n", issuer.index("commit(&st.tmem_full"))):]
    for bar in ("tmem_full[buf]", "empty[s]"):
        assert f"commit(&st.{bar})" in block and f"mbar_arrive(&st.{bar})" in block, bar
    for bar in ("empty[s]", "tmem_full[b]"):
        assert f"mbar_init(&st.{bar}, kMode == kBlock ? 2 : 1)" in text, bar


def test_bodies_of_the_grouped_gemms_read_with_plain_loads():
    """The same for the two forms whose kernels only call them."""
    for name, entry in (("gemm_sm100.cu", "void row_tiles("), ("gemm_wm.cuh", "void weights_on_m(")):
        text = source(name)
        body = braces(text, text.index(entry))
        assert "pdl_wait(" in body
        for word in ("__restrict__", "__ldg", "ld_nc16", ".nc"):
            assert word not in body, (name, word)


def test_what_is_read_before_the_wait_comes_past_l1():
    """The weights-on-M GEMM and the layer's block-scaled one copy the sort's table before their own griddepcontrol.wait. The sort is
    over by then, but only the wait covers lines of an earlier call's table that are still in L1."""
    for name, entry, tables in (("gemm_wm.cuh", "void weights_on_m(", ["offsets"]),
                                ("gemm_mx_sm100.cu", "__global__", ["offsets", "mtile_prefix"])):
        text = source(name)
        kernel = braces(text, text.index(entry))
        for table in tables:
            reads = re.findall(r"[\w ]*\(?\bp\." + table + r"\b", kernel)
            assert reads and all(r.endswith("ld_relaxed_gpu(p." + table) for r in reads), (name, reads)
    assert "ld.relaxed.gpu.global" in source("common.cuh")
    choice = braces(source("gemm_sm100.cu"), source("gemm_sm100.cu").index("bool weights_on_m_suit("))
    assert len(re.findall(r"ld_relaxed_gpu\(offsets \+", choice)) == len(re.findall(r"\boffsets\b", choice)) == 2


def test_roles_wait_for_the_kernel_before_before_they_wait_at_a_barrier():
    """A wait at a barrier gives up after a time that is meant for this kernel. Launched early, a role that has not yet waited for
    the kernel before would count that one's rest, however long it is held up, against it."""
    for name, entry in (("gemm_wm.cuh", "void weights_on_m("), ("gemm_mx_sm100.cu", "__global__")):
        text = source(name)
        kernel = braces(text, text.index(entry))
        roles = kernel[kernel.index("if (warp < 4) {"):]
        at = [m.start() for m in re.finditer(r"if \(warp == \d\)|else if constexpr \(kBlockMode\) \{\s*pdl_wait|"
                                             r"else \{\s*(?:ptx::setmaxnreg_inc<\w+>\(\);\s*)?pdl_wait", roles)] + [len(roles)]
        waits = 0
        for first, end in zip(at, at[1:]):
            role = roles[first:end]
            m = re.search(r"\bmbar_wait(_warp)?\(", role)
            if m:
                waits += 1
                assert "pdl_wait()" in role[:m.start()], (name, role[:200])
        assert waits == {"gemm_wm.cuh": 5, "gemm_mx_sm100.cu": 3}[name], name
        assert not re.search(r"\bmbar_wait(_warp)?\(", kernel[:kernel.index("if (warp < 4) {")]), name


def test_whole_warps_of_the_weights_on_m_form():
    """The same two rules there: the warp of the scale products and both epilogues wait together, and one lane arrives for a warp that
    has met."""
    text = source("gemm_wm.cuh")
    kernel = braces(text, text.index("void weights_on_m("))
    products = braces(kernel, kernel.index("else if (warp == 2)"))
    block = braces(kernel, kernel.index("else if constexpr (kBlockMode)", kernel.index("else if (warp == 2)")))
    plain = braces(kernel, kernel.index("else {", kernel.index(block) + len(block)))
    for role in (products, block, plain):
        assert "mbar_wait_warp(" in role and not re.search(r"\bmbar_wait\(", role), role[:100]
    for role, name in ((block, "auto release"), (plain, "auto release_tmem")):
        release = braces(role, role.index(name))
        assert release.index("__syncwarp()") < release.index("mbar_arrive")
        assert "mbar_arrive" not in role.replace(release, "")
    arrivals = [m.start() for m in re.finditer("mbar_arrive", products)]
    assert len(arrivals) == 1 and "__syncwarp()" in products[arrivals[0] - 100:arrivals[0]]


def test_kernels_before_an_early_gemm_start_it_after_their_own_wait():
    """An early grouped GEMM reads the sort's table and the weights before its own wait. That holds if it cannot start before the sort is
    over: a kernel that may stand right behind the sort lets its dependents start only after its wait, and so does an early GEMM
    itself. Others may stand between two of these, since they start behind the first: the re-quantisation pass and fc1's row tiles."""
    for name, kernels in (("permute.cu", ["scatter_rows_kernel", "scatter_quant_1x128_kernel"]),
                          ("quant_mx.cu", ["quant_rows_kernel", "tile_scales_kernel"])):
        text = source(name)
        for kernel in kernels:
            body = braces(text, text.index(kernel + "("))
            assert re.match(r"{\s*pdl_wait\(\);\s*pdl_launch\(\);", body) and body.count("pdl_") == 2, kernel
    wm = source("gemm_wm.cuh")
    wm = braces(wm, wm.index("void weights_on_m("))
    assert re.findall(r"if constexpr \((!?kEarly)\) pdl_launch\(\)", wm) == ["!kEarly", "kEarly", "kEarly"]
    assert len(re.findall(r"pdl_wait\(\);\s*if constexpr \(kEarly\) pdl_launch\(\)", wm)) == 2 and wm.count("pdl_launch()") == 3
    mx = source("gemm_mx_sm100.cu")
    mx = braces(mx, mx.index("__global__"))
    assert re.findall(r"if \((!?p\.early)\) pdl_launch\(\)", mx) == ["!p.early", "p.early"] and mx.count("pdl_launch()") == 2
    assert len(re.findall(r"pdl_wait\(\);\s*if \(p\.early\) pdl_launch\(\)", mx)) == 1
