"""CPU checks of rules that the CUDA sources keep and that no compiler checks."""
import glob
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ghostsuite_b200", "csrc")


def _sources():
    """``{file name: text}`` without comments."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = open(path).read()
        out[os.path.basename(path)] = re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))
    return out


def _body(text, start):
    """``text`` from the first brace at or after ``start`` to the one that closes it."""
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError("unbalanced braces")


def _kernels(text):
    """``(name, parameters, body)`` of every ``__global__`` function that is defined in ``text``."""
    for m in re.finditer(r"__global__\b", text):
        head = re.compile(r"\b(\w+_kernel)\s*\(([^{;]*)\)\s*\{").search(text, m.end())
        yield head.group(1), head.group(2), _body(text, head.end() - 1)


def test_kernels_that_start_early_read_with_ordinary_loads():
    """A kernel launched with programmatic stream order lives while the one ahead of it still writes, so its
    loads must not go through the read-only path (``ld.global.nc``: memory that nobody writes while the
    kernel lives)."""
    early = 0
    for name, text in _sources().items():
        for kernel, params, body in _kernels(text):
            if "stream_order()" in body:
                early += 1
                assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", params), f"{name}: {kernel}"
        if name == "embedding.cu":       # the rows of the join, which come up behind everything that it reads
            for m in re.finditer(r"struct EmbOct<\w+>", text):
                text = text.replace(_body(text, m.end()), "{" + " " * (len(_body(text, m.end())) - 2) + "}")
        if name == "proj_extras.cu":     # rows off vector boundaries: their kernel is launched in plain order
            assert "if constexpr (VEC) stream_order();" in text
            calls = re.findall(r"sim_launch\(proj_similarity_kernel<[^>]*, (\w+), \w+>, (\w+),", text)
            assert len(calls) == 4 and all(vec == starts_early for vec, starts_early in calls)
            unaligned = "for (int e = 0; e < 8; ++e) v[e] = ok && k + e < d ? __ldg(row + k + e) : 0.f;"
            assert text.count(unaligned) == 1
            text = text.replace(unaligned, "")
        assert "__ldg(" not in text and "ld.global.nc" not in text, name
    assert early >= 20


def test_a_type_is_defined_once():
    """The translation units pass structures to each other by reference: a second definition of one that is
    changed later would still link."""
    where = {}
    for name, text in _sources().items():
        for m in re.finditer(r"\b(?:struct|class|union)\s+(\w+(?:<[^<>{};]*>)?)\s*(?::[^{;]*)?\{", text):
            where.setdefault(m.group(1), []).append(name)
    assert len(where) > 20
    assert {k: v for k, v in where.items() if len(v) > 1} == {}


def test_every_header_makes_the_library_stale():
    from ghostsuite_b200 import build
    headers = {os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h"))}
    assert headers <= set(build.HEADERS) and "launch_rules.h" in build.HEADERS[-2:]


def test_alignment_slack_of_the_shared_memory_is_not_used():
    """Dynamic shared memory is asked for with 1024 bytes to spare, by which its start is rounded up: no piece
    may be placed as if the start were aligned already."""
    placed = 0
    for name, text in _sources().items():
        for m in re.finditer(r"\bsmem \+ [^;,]*", text):
            placed += 1
            assert "1024" not in m.group(0), f"{name}: {m.group(0)}"
    assert placed > 20


def test_words_of_an_embedding_table_are_counted_in_64_bits():
    """A table may have up to 2^31 - 1 rows; its counts and the totals before them are more words than that."""
    sums = [line for line in _sources()["embedding.cu"].splitlines() if "vocab" in line and re.search(r"kEmbTotals \+|\+ kEmbTotals", line)]
    assert len(sums) >= 4
    for line in sums:
        assert re.search(r"static_cast<(long long|size_t)>\(\w*\.?vocab\)", line), line


def test_barriers_of_whole_warps_bring_the_warp_together():
    """``bar`` and ``barrier.cluster.*.aligned`` must be entered by all lanes of a warp at once: they stand in functions that
    see to it, and nowhere else."""
    sources = _sources()
    for name in ("named_bar_and", "named_bar_sync", "cluster_sync_all"):
        text = sources["sm100_ptx.cuh"]
        body = _body(text, re.search(r"\b%s\([^)]*\) \{" % name, text).start())
        assert "__syncwarp();" in body[:body.index("asm")], name
        sources["sm100_ptx.cuh"] = text.replace(body, "{}")
    for name, text in sources.items():
        assert not re.search(r"\bbar\.(sync|red|arrive)|\bbarrier\.cluster", text), name


def test_a_count_that_the_driver_refused_is_not_kept():
    """How many clusters are resident is asked once per kernel and device, unless the question failed."""
    text = _sources()["gradproj.cu"]
    body = _body(text, text.index("gradproj_resident(int ranks"))
    refused = _body(body, body.index("cudaOccupancyMaxActiveClusters"))
    assert "return 0;" in refused and "store" not in refused
    assert body.index(refused) < body.index("slot.store(")


def _answers(tmp_path, calls):
    """What the rules of launch_rules.h answer to ``calls`` (C++ expressions), each as a number."""
    src, exe = tmp_path / "rules.cpp", tmp_path / "rules"
    body = "".join(f'  std::printf("%.17g\\n", static_cast<double>(gb::{c}));\n' for c in calls)
    src.write_text('#include <cstdio>\n#include "launch_rules.h"\nint main() {\n' + body + "}\n")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, f"ended by signal {-done.returncode}"
    return [float(x) for x in done.stdout.split()]


def test_copies_of_projection_operands(tmp_path):
    """An empty call is answered too (the kernel's own check refuses it), and so is one on a device that was refused."""
    empty = [f"gradproj_copies({b}, {t}, 65, 40, false, {ready}, {sms})"
             for b, t in ((0, 5), (3, 0), (0, 0)) for ready in ("false", "true") for sms in (148, 0, -3)]
    assert set(_answers(tmp_path, empty)) == {0}
    # calls that are named beside the rule, each on its faster side
    measured = {"26, 471, 9408, 795, true, false": 1, "10, 30, 6912, 2579, true, false": 1, "28, 5, 3957, 9063, false, false": 1,
                "32, 3000, 1001, 2003, false, false": 0, "4, 9, 64, 64, true, true": 0}
    assert _answers(tmp_path, [f"gradproj_copies({c}, 148)" for c in measured]) == list(measured.values())


def test_splits_of_a_train_gradient(tmp_path):
    """(tiles, CTAs, row blocks, time of one, cost of an addition, elements, float32) of measured calls on 148 SMs: what a
    merge costs counts in the time of a block of the kernel that is meant."""
    single = {"65, 148, 47, 0.35, 12, 1600. * 1200, false": 1, "65, 148, 64, 0.35, 12, 1600. * 1200, false": 1,
              "65, 148, 128, 0.35, 12, 1600. * 1200, false": 2, "45, 148, 32, 0.35, 12, 1152. * 1152, false": 1}
    pairs = {"36, 74, 64, 0.65, 6, 3072. * 768, false": 2}
    assert _answers(tmp_path, [f"pick_k_splits({c})" for c in {**single, **pairs}]) == [*single.values(), *pairs.values()]
    # few tiles are shared, one block is not
    few, one = _answers(tmp_path, ["pick_k_splits(1, 148, 64, 0.35, 12, 128. * 128, false)", "pick_k_splits(1, 148, 1, 0.35, 12, 128. * 128, false)"])
    assert few > 4 and one == 1


def test_clusters_of_gram_tiles_and_few_row_layers(tmp_path):
    """Sizes on either side of the lines, on 148 SMs with as many clusters resident as fit: (tiles, K steps), and (pairs of groups, tiles a
    pair, blocks of the gradient, train rows, columns of the operands)."""
    gram = {"2, 163": 8, "8, 48": 8, "40, 30": 3, "32, 15": 4, "1, 11": 1, "75, 400": 1, "3, 1": 1}
    answers = _answers(tmp_path, [f"gram_cluster({c}, 148, [](int r) {{ return 148 / r; }})" for c in gram])
    assert answers == list(gram.values())
    assert _answers(tmp_path, ["gram_cluster(2, 163, 148, [](int) { return 0; })"]) == [1]       # a refused question: no cluster
    small = {"2, 1, 0, 4, 108, 27072": 8, "4, 1, 0, 8, 8192, 260": 8, "2, 8, 0, 128, 2048, 1024": 1, "1, 1, 9384, 2, 768, 50000": 1, "3, 1, 0, 4, 64, 64": 1,
             "200, 1, 0, 200, 20000, 20000": 1}
    assert _answers(tmp_path, [f"small_cluster({c}, 148)" for c in small]) == list(small.values())
