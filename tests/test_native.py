"""Host code of the library that no entry point reaches by itself, compiled into small C++ programs: index arithmetic of the kernels
over its whole range, and calls of the CUDA runtime or of the C library that fail (fakes of those calls; no GPU is involved)."""
import os
import subprocess

import pytest

import harness
from aspen_b200 import api, cfgs

from test_gpu_shapes import RANGE_SHAPES, SPLIT_SHAPES

HERE = os.path.dirname(os.path.abspath(__file__))
LIBDIR = os.path.join(os.path.dirname(HERE), "aspen_b200")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def build(name, workdir, *flags):
    exe = os.path.join(workdir, name)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", os.path.join(HERE, "native", name + ".cpp"), "-o", exe, *flags], check=True)
    return exe


def passes(exe, *args, timeout=20):
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=timeout)
    assert r.returncode == 0, r.stdout + r.stderr


def test_division_by_multiplication_is_exact(workdir):
    passes(build("index_div", workdir))


@pytest.fixture(scope="module")
def host_copy(tmp_path_factory):
    return build("host_copy", str(tmp_path_factory.mktemp("native")), "-I", CUDA_INCLUDE, "-rdynamic", "-lpthread", "-ldl")


@pytest.mark.parametrize("fault", [(), ("event", "1"), ("event", "16"), ("ring",), ("thread", "1"), ("thread", "2"), ("resident",)], ids=" ".join)
def test_results_arrive_whatever_part_of_the_copy_team_cannot_be_made(host_copy, fault):
    passes(host_copy, *fault)


def test_a_graph_is_the_same_with_any_number_of_threads(workdir):
    api.lib()
    exe = build("few_threads", workdir, "-rdynamic", f"-L{LIBDIR}", "-laspen_b200", f"-Wl,-rpath,{LIBDIR}", "-lpthread", "-ldl")
    cfg, _ = harness.prepare("custom", workdir)
    files = [os.path.join(workdir, f"threads_{n}.nasm") for n in (1, 3, 1000)]
    for n, f in zip((1, 3, 1000), files):
        passes(exe, str(n), cfg, "16", f)
    graphs = [open(f, "rb").read() for f in files]
    assert graphs[0] == graphs[1] == graphs[2] and len(graphs[0]) > 100000


@pytest.mark.parametrize("seed", ["1", "2", "3"])
def test_every_worker_warp_leaves_whichever_waits_give_up(seed, workdir):
    passes(build("worker_loop", workdir, "-lpthread"), seed)


def operand_forms(workdir, text, seq=0):
    api.lib()
    exe = build("operand_forms", workdir, f"-L{LIBDIR}", "-laspen_b200", f"-Wl,-rpath,{LIBDIR}")
    cfg = os.path.join(workdir, "forms.cfg")
    with open(cfg, "w") as f:
        f.write(text)
    r = subprocess.run([exe, cfg, str(seq)], capture_output=True, text=True, check=True).stdout
    return [tuple(int(v) for v in line.split()[1:]) for line in r.split("\n")[1:-1]]


def test_layers_of_any_channel_count_have_a_form_for_the_tensor_cores(workdir):
    """300 x 300 image, 48- and 24-channel convolutions: every contraction reaches the tensor cores, the taps of the weights in whole
    chunks of 32; a second convolution on the image goes tap by tap, and what an im2col map cannot hold does not go at all."""
    conv = "[convolutional]\nfilters={}\nsize={}\nstride={}\npad={}\n{}\n"
    forms = operand_forms(workdir, "[net]\nheight=300\nwidth=300\nchannels=3\n\n" + conv.format(48, 7, 2, 3, "") + conv.format(24, 3, 1, 1, "") +
                          conv.format(64, 1, 1, 0, "") + conv.format(8, 1, 2, 0, "") + conv.format(8, 3, 1, 1, "parent=-5\n") + conv.format(8, 3, 1, 3, "") +
                          conv.format(8, 3, 9, 1, "") + "[connected]\noutput=10\n\n")
    assert forms == [(2, 1, 7 * 32), (2, 0, 9 * 64), (1, 0, 0), (2, 0, 64), (2, 0, 9 * 32), (0, 0, 0), (0, 0, 0), (1, 0, 0)]


@pytest.mark.parametrize("heads,d,seq,form", [(2, 64, 100, 1), (2, 160, 100, 3), (4, 48, 512, 3), (4, 40, 100, 0), (2, 64, 513, 0)])   # 0: not
def test_attention_heads_of_a_multiple_of_four_have_a_form_for_the_tensor_cores(heads, d, seq, form, workdir):
    text, _ = cfgs.transformer(1, d, heads, d, pre_ln=False, masked=False, act="gelu")
    forms = operand_forms(workdir, text, seq)
    assert [f[0] for f in forms[:6]] == [1, 1, 1, form, 1 if d // heads % 4 == 0 else 0, 1]


@pytest.mark.parametrize("batch,seq,d,heads", [(2, 600, 256, 4), (8, 128, 120, 12)])
def test_the_plan_spreads_layers_that_do_not_run_on_the_tensor_cores(batch, seq, d, heads, workdir):
    """Scores of 600 keys, or of heads of 10: fp32 blocks one after the other on an SM, so no SM may be left with the work of several
    (costed as tensor-core tiles they were 40 and 96 tiles for 148 SMs)."""
    api.lib()
    text, _ = cfgs.transformer(1, d, heads, d, pre_ln=False, masked=False, act="gelu")
    exe = build("plan_tiles", workdir, f"-L{LIBDIR}", "-laspen_b200", f"-Wl,-rpath,{LIBDIR}")
    cfg = os.path.join(workdir, "plan.cfg")
    with open(cfg, "w") as f:
        f.write(text)
    r = subprocess.run([exe, cfg, str(batch), str(seq), "148"], capture_output=True, text=True, check=True).stdout
    layers = [(line.split()[0], [int(v) for v in line.split()[1:]]) for line in r.split("\n")[:-1]]
    th, tw, tiles = next(v for t, v in layers if "K_ATTENTION" in t)
    assert tiles >= 148 and th == seq


@pytest.mark.parametrize("name,batch,seq,workers", [("tiny_cnn", 3, 0, 148), ("resnet50", 2, 0, 148), ("bert_base", 1, 37, 148), ("tiny_transformer", 2, 16, 1), ("custom", 5, 0, 7)])
@pytest.mark.parametrize("precision", [0, 1])
def test_a_launch_hands_out_every_tile_once_behind_its_parents(name, batch, seq, workers, precision, workdir):
    """In the fp32 mode with the lists of layers whose k several tiles share, too (ResNet-50 and BERT have such layers at these sizes)."""
    api.lib()
    exe = build("claim_order", workdir, f"-L{LIBDIR}", "-laspen_b200", f"-Wl,-rpath,{LIBDIR}")
    cfg, _ = harness.prepare(name, workdir)
    r = subprocess.run([exe, cfg, str(batch), str(seq), str(workers), str(precision)], capture_output=True, text=True, timeout=20)
    assert r.returncode == 0, r.stdout + r.stderr
    assert (int(r.stdout) > 0) == (precision == 1 and name in ("resnet50", "bert_base"))


def test_shapes_that_test_the_split_kernels_run_them(workdir):
    """Of the allocation-free matmul, on the 148 SMs of a B200: every instance (block of 128 or 64 rows, 4, 2 or 1 values a load)."""
    exe = build("matmul_pick", workdir)
    seen = set()
    for n, k, m, kernel in SPLIT_SHAPES + RANGE_SHAPES:
        values = next(v for v in (4, 2, 1) if k % v == 0)
        picked = subprocess.run([exe, *(str(v) for v in (n, k, m, 148, values))], capture_output=True, text=True, check=True).stdout
        assert picked == kernel, (n, k, m)
        seen.add((kernel, values))
    assert len(seen) == 6


@pytest.mark.parametrize("n,k,m,values,us", [(446, 167, 2114, 1, (31.6, 37.7)), (727, 178, 1253, 2, (27.6, 31.4)), (395, 23, 2300, 1, (18.9, 25.5)), (3566, 143, 512, 1, (40.6, 56.5)),
                                             (709, 232, 1421, 4, (36.8, 39.1))])
def test_short_sums_of_many_outputs_run_in_large_blocks(n, k, m, values, us, workdir):
    """us: of a call on a B200, in 128 x 64 blocks and in 32 x 32 ones."""
    assert subprocess.run([build("matmul_pick", workdir), *(str(v) for v in (n, k, m, 148, values))], capture_output=True, text=True, check=True).stdout == "fma 128x64"


def test_calls_that_run_at_once_have_numbers_of_their_own(workdir):
    passes(build("call_slots", workdir, "-lpthread"), timeout=60)


def test_sets_of_graphs_that_are_run_in_turn_are_kept(workdir):
    passes(build("recent_sets", workdir))


def test_a_launch_of_several_graphs_has_the_small_ones_done_first(workdir):
    api.lib()
    passes(build("merge_claims", workdir, f"-L{LIBDIR}", "-laspen_b200", f"-Wl,-rpath,{LIBDIR}"))
