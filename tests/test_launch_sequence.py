"""Which kernels a call launches, without a GPU: the library's sources compiled over a CUDA runtime that records
launches instead of making them (launch_recorder.cpp)."""
import ctypes
import os
import re
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

from gevva_b200 import build
from gevva_b200 import feedforward as ff
from gevva_b200 import runtime as rt

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which(build.NVCC)
STREAM, AUX_STREAM = 64, 65
ADDRESS = 4096  # stands for every pointer that the recording runtime does not follow


def kernel_name(mangled):
    """The function's own name, followed by <0> or <1> where its first template argument is a bool."""
    for digits in re.finditer(r"\d+", mangled):
        for start in range(digits.start(), digits.end()):
            length = int(mangled[start : digits.end()])
            name = mangled[digits.end() : digits.end() + length]
            if len(name) == length and name.endswith("_kernel"):
                flag = re.match(r"ILb([01])E", mangled[digits.end() + length :])
                return name + (f"<{flag[1]}>" if flag else "")
    return mangled


class Recorder:
    def __init__(self, path):
        self.lib = lib = ctypes.CDLL(path)
        lib.recorder_take_log.restype = ctypes.c_char_p
        vp, i32 = ctypes.c_void_p, ctypes.c_int
        lib.gevva_moe_create.argtypes = [ctypes.POINTER(vp), ctypes.POINTER(rt._Weights), i32, vp, ctypes.POINTER(rt._Options)]
        lib.gevva_moe_destroy.argtypes = [vp]
        lib.gevva_moe_launch_stages.argtypes = [vp, vp, vp, vp, vp, i32, ctypes.c_uint, vp]
        lib.gevva_dense_create.argtypes = [ctypes.POINTER(vp), ctypes.POINTER(ff._DenseWeights), i32]
        lib.gevva_dense_destroy.argtypes = [vp]
        lib.gevva_dense_launch.argtypes = [vp, vp, vp, i32, vp]
        lib.gevva_dense_status_word.argtypes = lib.gevva_moe_status_word.argtypes = [vp]
        lib.gevva_dense_status_word.restype = lib.gevva_moe_status_word.restype = ctypes.c_size_t
        lib.gevva_ff_layer_launch.argtypes = [ctypes.POINTER(ff._Layer), vp, vp, vp, i32, vp, vp]

    def runner(self, max_tokens, flags=0):
        handle = ctypes.c_void_p()
        assert self.lib.gevva_moe_create(ctypes.byref(handle), ctypes.byref(rt._Weights(*[ADDRESS] * 8)), max_tokens, None,
                                         ctypes.byref(rt._Options(flags))) == 0
        self.launches()
        return handle

    def dense(self, max_tokens):
        handle = ctypes.c_void_p()
        assert self.lib.gevva_dense_create(ctypes.byref(handle), ctypes.byref(ff._DenseWeights(ADDRESS, ADDRESS, 1, 1, 1)),
                                           max_tokens) == 0
        self.launches()
        return handle

    def launches(self):
        """The launches since the last call: dicts with the kernel's name and the launch's attributes."""
        out = []
        for line in self.lib.recorder_take_log().decode().splitlines():
            mangled, rest = line.split(" ", 1)
            out.append({key: int(value) for key, value in re.findall(r"(\w+)=(\d+)", rest)})
            out[-1]["kernel"] = kernel_name(mangled)
        return out

    def layer(self, runner, tokens, stages=rt.STAGE_ALL):
        assert self.lib.gevva_moe_launch_stages(runner, ADDRESS, ADDRESS, ADDRESS, ADDRESS, tokens, stages, STREAM) == 0
        return self.launches()


@pytest.fixture(scope="module")
def recorder(tmp_path_factory):
    if NVCC is None:
        pytest.skip("needs nvcc")
    folder = tmp_path_factory.mktemp("recorder")

    def compile_one(source):
        target = str(folder / (os.path.splitext(os.path.basename(source))[0] + ".o"))
        # PTX only: the device code is not run
        subprocess.run([NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=compute_100a", "-Xcompiler", "-fPIC",
                        "-c", "-o", target, source], check=True, capture_output=True)
        return target

    sources = [os.path.join(build.CSRC, s) for s in build.SOURCES if s.endswith(".cu")]
    with ThreadPoolExecutor(os.cpu_count()) as pool:
        objects = list(pool.map(compile_one, sources + [os.path.join(ROOT, "tests", "launch_recorder.cpp")]))
    library = str(folder / "librecorder.so")
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", library] + objects + ["-ldl"], check=True, capture_output=True)
    return Recorder(library)


def kernels(launches):
    return [launch["kernel"] for launch in launches]


@pytest.mark.parametrize("flags", [0, rt.OPTION_PAIRS, rt.OPTION_W13_PAIRS])
@pytest.mark.parametrize("tokens", [1, 64, 128, 129, 296, 297, 640, 641])
def test_kernels_of_a_layer(recorder, flags, tokens):
    """The pair options are for batches of more than 128 tokens; smaller ones run as without them."""
    runner = recorder.runner(1024, flags)
    got = kernels(recorder.layer(runner, tokens))
    plain_front = ["route_sort_fused_kernel", "quantize_input_kernel<1>"]
    if tokens <= 128 or (flags == 0 and tokens <= 296):
        assert got == ["stream_experts_kernel<1>", "reduce_routes_kernel<0>"]
    elif flags == 0 and tokens <= 640:
        assert got == plain_front + ["stream_experts_kernel<0>", "reduce_routes_kernel<0>"]
    elif flags == rt.OPTION_PAIRS:
        assert got == plain_front + ["grouped_nvfp4_gemm_pair_kernel"] * 2 + ["reduce_routes_kernel<0>"]
    else:
        assert got == plain_front + ["w13_geglu_pair_kernel", "grouped_down_kernel", "reduce_routes_kernel<1>"]
    recorder.lib.gevva_moe_destroy(runner)


@pytest.mark.parametrize("tokens", [129, 641, 1024])
def test_switches_give_the_one_cta_kernels(recorder, monkeypatch, tokens):
    """What the other forms of the two GEMMs are compared with bit by bit."""
    monkeypatch.setenv("GEVVA_MOE_DECODE_MERGED", "0")
    monkeypatch.setenv("GEVVA_MOE_W13_PAIRS", "0")
    runner = recorder.runner(1024)
    assert kernels(recorder.layer(runner, tokens))[2:4] == ["grouped_nvfp4_gemm_kernel", "grouped_down_kernel"]
    recorder.lib.gevva_moe_destroy(runner)


def layer_launch(recorder, runner, dense, tokens, router_weight=ADDRESS, workspace=ADDRESS):
    layer = ff._Layer(*[ADDRESS] * 9, runner, dense)
    layer.router_weight = router_weight
    return recorder.lib.gevva_ff_layer_launch(ctypes.byref(layer), ADDRESS, ADDRESS, workspace, tokens, STREAM, AUX_STREAM)


def test_feed_forward_layer_launches(recorder):
    runner, dense = recorder.runner(64), recorder.dense(64)
    assert layer_launch(recorder, runner, dense, 64) == 0
    launches = recorder.launches()
    assert kernels([l for l in launches if l["stream"] == AUX_STREAM]) == [
        "fp8_quantize_rows_kernel", "grouped_nvfp4_gemm_kernel", "gelu_quantize_fp8_kernel", "grouped_nvfp4_gemm_kernel"]
    assert kernels([l for l in launches if l["stream"] == STREAM]) == [
        "ff_prepare_kernel", "route_project_kernel<0>", "stream_experts_kernel<1>", "ff_finalize_kernel"]


@pytest.mark.parametrize("tokens,share", [(40, 16), (128, 16), (129, 22), (640, 33), (641, 0)])
@pytest.mark.parametrize("flags,merged", [(0, "1"), (rt.OPTION_PAIRS, "1"), (rt.OPTION_W13_PAIRS, "1"), (0, "0")])
def test_sms_of_the_two_sides_of_a_layer(recorder, monkeypatch, flags, merged, tokens, share):
    """Above 128 tokens the dense MLP gets SMs of its own only where the experts stream; else both sides take all of them."""
    monkeypatch.setenv("GEVVA_MOE_DECODE_MERGED", merged)
    runner, dense = recorder.runner(1024, flags), recorder.dense(1024)
    assert layer_launch(recorder, runner, dense, tokens) == 0
    launches = recorder.launches()
    gemms = lambda stream: [l for l in launches if l["stream"] == stream and re.match("stream|grouped|w13|dense_fp8", l["kernel"])]
    if tokens > 128 and (flags or merged == "0"):
        share = 0
    assert {l["grid"] for l in gemms(STREAM)} == {148 - share}
    assert {(l["kernel"], l["grid"]) for l in gemms(AUX_STREAM)} == (
        {("grouped_nvfp4_gemm_kernel", share)} if share else {("dense_fp8_pair_kernel", 148)})


@pytest.mark.parametrize("offset,last", [(0, "dense_fp8_pair_kernel"), (16, "grouped_nvfp4_gemm_kernel"),
                                         (32, "dense_fp8_pair_kernel"), (48, "grouped_nvfp4_gemm_kernel")])
def test_dense_outputs_between_32_byte_lines(recorder, offset, last):
    """The pair kernel stores 32 bytes at a time: into an output that is aligned to 16 only, the one-CTA kernel stores."""
    dense = recorder.dense(64)
    assert recorder.lib.gevva_dense_launch(dense, ADDRESS, ADDRESS + offset, 64, STREAM) == 0
    assert kernels(recorder.launches()) == ["fp8_quantize_rows_kernel", "dense_fp8_pair_kernel", "gelu_quantize_fp8_kernel", last]


@pytest.mark.parametrize("tokens,few", [(1, True), (2, True), (3, False)])
def test_dense_mlp_of_a_few_tokens(recorder, tokens, few):
    dense = recorder.dense(64)
    assert recorder.lib.gevva_dense_launch(dense, ADDRESS, ADDRESS + 16, tokens, STREAM) == 0
    got = kernels(recorder.launches())
    want = (["dense_few_gate_up_kernel", "dense_few_down_kernel"] if few else
            ["fp8_quantize_rows_kernel", "dense_fp8_pair_kernel", "gelu_quantize_fp8_kernel", "grouped_nvfp4_gemm_kernel"])
    assert len(got) == len(want) and all(name.endswith(end) for name, end in zip(got, want))


@pytest.mark.parametrize("offset", [0, 16])
def test_dense_waits_report_where_they_are_read(recorder, offset):
    """A wait of the dense MLP that runs out is reported into a word that a status call reads: its own, in a layer the experts'."""
    runner, dense = recorder.runner(1024), recorder.dense(1024)
    assert recorder.lib.gevva_dense_launch(dense, ADDRESS, ADDRESS + offset, 600, STREAM) == 0
    words = [l["status"] for l in recorder.launches() if l["status"]]
    assert len(words) == 2 and set(words) == {recorder.lib.gevva_dense_status_word(dense)}
    assert recorder.lib.gevva_dense_launch(dense, ADDRESS, ADDRESS + offset, 2, STREAM) == 0
    assert [l["status"] for l in recorder.launches()] == [recorder.lib.gevva_dense_status_word(dense)] * 2
    for tokens in (1, 2, 40, 600, 1000):
        assert layer_launch(recorder, runner, dense, tokens) == 0
        words = [l["status"] for l in recorder.launches() if l["stream"] == AUX_STREAM and l["status"]]
        assert len(words) == 2 and set(words) == {recorder.lib.gevva_moe_status_word(runner)}


@pytest.mark.parametrize("in_offset,out_offset", [(8, 0), (2, 0), (0, 8), (0, 2)])
def test_dense_refuses_unaligned_rows(recorder, in_offset, out_offset):
    dense = recorder.dense(64)
    assert recorder.lib.gevva_dense_launch(dense, ADDRESS + in_offset, ADDRESS + out_offset, 64, STREAM) == -3
    assert recorder.launches() == []


@pytest.mark.parametrize("capacity,dense_capacity,tokens,router_weight", [(4, 64, 5, ADDRESS), (64, 4, 5, ADDRESS),
                                                                         (64, 64, 0, ADDRESS), (64, 64, 5, ADDRESS + 8)])
def test_feed_forward_layer_refuses_before_it_launches(recorder, capacity, dense_capacity, tokens, router_weight):
    """A call that one of its parts would refuse launches nothing: neither of the parts in front of it, on either stream."""
    runner, dense = recorder.runner(capacity), recorder.dense(dense_capacity)
    assert layer_launch(recorder, runner, dense, tokens, router_weight) == -3  # GEVVA_MOE_BAD_ARGUMENT
    assert recorder.launches() == []


@pytest.mark.parametrize("device,sms", [(0, 148), (1, 74)])
def test_prepare_takes_three_ctas_of_each_sm_that_there_is(recorder, device, sms):
    """A CTA a row up to as many as run at once on the current device, then so many CTAs that take row after row."""
    recorder.lib.recorder_set_device(device, sms)
    try:
        for rows in (1, 3 * sms, 3 * sms + 1, 4096):
            assert recorder.lib.gevva_ff_prepare(*[ctypes.c_void_p(ADDRESS)] * 7, rows, ctypes.c_void_p(STREAM)) == 0
            (launch,) = recorder.launches()
            assert (launch["kernel"], launch["grid"]) == (("ff_prepare_kernel", rows) if rows <= 3 * sms else ("ff_prepare_rows_kernel", 3 * sms))
    finally:
        recorder.lib.recorder_set_device(0, 148)


class _Cuda:
    """What forward() checks of a tensor."""
    is_cuda = True
    device = "cuda:0"

    def __init__(self, shape, dtype, contiguous=True):
        self.shape, self.dtype, self._contiguous = torch.Size(shape), dtype, contiguous

    def is_contiguous(self):
        return self._contiguous


@pytest.mark.parametrize("router_w,expert_scale", [
    (_Cuda((128, 2816), torch.uint8), None), (_Cuda((128, 2816), torch.float32), None),
    (_Cuda((64, 2816), torch.bfloat16), None), (_Cuda((128, 2816), torch.bfloat16, False), None),
    (None, _Cuda((128,), torch.float32)), (None, _Cuda((64,), torch.bfloat16))])
def test_feed_forward_layer_checks_its_router(router_w, expert_scale):
    """forward() hands addresses to one native call, so what route_project() would refuse it has to refuse itself."""
    router_w = router_w or _Cuda((128, 2816), torch.bfloat16)
    expert_scale = expert_scale or _Cuda((128,), torch.bfloat16)
    layer = ff.FeedForwardLayer(*[None] * 3, router_w, expert_scale, *[None] * 6)
    with pytest.raises(ValueError, match="router_weight|expert_scale"):
        layer.forward(_Cuda((3, 2816), torch.bfloat16))
