"""Which kernel a call of few rows goes to (csrc/capi.cc, csrc/skinny_stream.cu), against the CUDA runtime that runs nothing
and records every launch (fake_cuda.c)."""
import pytest

from test_many_row_host_cpu import fake  # noqa: F401  (a fixture)


def _kernel(log):
    return [next((k for k in ("SkinnyGemmStreamKernel", "SkinnyGemm") if k in line), line.split()[0]) for line in log]


@pytest.mark.parametrize("dtype", ["BF16", "FP8", "U8"])
def test_routes(fake, dtype):  # noqa: F811
    """Copies need rows of 16 bytes (NVFP4: 8) and K in eights; a pinned geometry, and a map that cannot be made, are the
    general kernels'."""
    narrow = 192 if dtype == "U8" else 264 if dtype == "FP8" else 260
    out = fake(f"""
        h = gemm([1], [256])
        r = [run_gemm(h, {dtype}, m, 512, [[256]]) for m in (1, 8)]
        r += [run_gemm(h, {dtype}, 2, 516, [[256]]), run_gemm(gemm([1], [{narrow}]), {dtype}, 2, 512, [[{narrow}]]),
              run_gemm(gemm([1], [256], plan="wn=1,wk=2,cluster=1"), {dtype}, 2, 512, [[256]]),
              run_gemm(gemm([1], [256], stream_plan="0"), {dtype}, 2, 512, [[256]])]
        fake.fake_refuse_encode(1)
        r.append(run_gemm(h, {dtype}, 2, 512, [[256]]))
        fake.fake_refuse_encode(0)
        os.environ["QFG_PLAN"] = "wn=1,wk=2,cluster=1"
        r.append(run_gemm(gemm([1], [256]), {dtype}, 2, 512, [[256]]))
        print(json.dumps(r))
        """)
    for code, message, _ in out:
        assert code == 0, message
    assert [_kernel(log) for _, _, log in out] == [["SkinnyGemmStreamKernel"]] * 2 + [["SkinnyGemm"]] * 6


@pytest.mark.parametrize("dtype", ["BF16", "FP8", "U8"])
def test_shared_expert_in_passes_of_eight(fake, dtype):  # noqa: F811
    out = fake(f"""
        s = shared(pdl_wait=1)
        calls = fake.fake_setup_calls()
        fake.fake_refuse_setup(1)
        r = [run_shared(s, {dtype}, m, 256, 128) for m in (3, 16)]
        general = shared(stream_plan="0", dense_rows=0, pdl_wait=1)
        r.append(run_shared(general, {dtype}, 20, 256, 128))
        fake.fake_device(1)
        print(json.dumps([r, run_shared(s, {dtype}, 3, 256, 128), calls == fake.fake_setup_calls()]))
        """)
    (few, two_passes, general), other_device, no_setup = out
    assert general[0] == 0 and _kernel(general[2]) == ["SkinnyGemm"] * 3
    assert few[0] == two_passes[0] == 0 and no_setup
    assert _kernel(few[2]) == ["SkinnyGemmStreamKernel"] and _kernel(two_passes[2]) == ["SkinnyGemmStreamKernel"] * 2
    assert all(line.endswith("pdl=1") for line in few[2] + two_passes[2])
    assert other_device[0] != 0


@pytest.mark.parametrize("dtype,k,widths", [("BF16", 5120, [5120]), ("FP8", 6144, [2560]), ("U8", 5120, [17408, 17408]), ("U8", 17408, [5120]), ("BF16", 516, [256])])
def test_the_described_plan_is_the_launched_one(fake, dtype, k, widths):  # noqa: F811
    out = fake(f"""
        fake.fake_resident(148)
        h = gemm([1] * {len(widths)}, {widths})
        buf = ctypes.create_string_buffer(512)
        w = (L.Tensor2D * {len(widths)})(*[L.Tensor2D(P, {dtype}, {k}, cols({dtype}, n)) for n in {widths}])
        assert lib.qfg_skinny_gemm_describe(h, {k}, w, {len(widths)}, buf, 512) == 0
        pinned = L.plan_describe({dtype}, {k}, {widths}, spec="wn=1,wk=2,cluster=1")
        print(json.dumps([run_gemm(h, {dtype}, 1, {k}, [[n] for n in {widths}]), L.plan_describe({dtype}, {k}, {widths}), pinned, buf.value.decode()]))
        """)
    (code, message, log), plan, pinned, described = out
    assert code == 0, message
    keys = ("width", "wk", "teams", "cluster", "tail")
    assert "stream=" + "/".join(str(plan[f"stream_{key}"]) for key in keys) in described
    assert pinned["stream_width"] == 0
    if k % 8:
        assert plan["stream_width"] == 0 and _kernel(log) == ["SkinnyGemm"]
        return
    assert _kernel(log) == ["SkinnyGemmStreamKernel"]
    columns = {"BF16": 8, "FP8": 16, "U8": 128}[dtype] * plan["stream_width"]
    tiles = sum(-(-n // columns) for n in widths)
    wide = -(-columns // {"BF16": 64, "FP8": 128, "U8": 128}[dtype])
    threads = 32 * (plan["stream_wk"] * plan["stream_teams"] * wide + 1)
    assert f"grid={tiles},{plan['stream_cluster']} threads={threads} " in log[0], (plan, log)


@pytest.mark.parametrize("resident,clusters", [(132, True), (1, False)])
def test_clusters_that_the_device_holds(fake, resident, clusters):  # noqa: F811
    # K short enough for eight rows of x in one CTA (16384 would take 256 KB): without clusters the kernel is still the one
    out = fake(f"""
        fake.fake_resident({resident})
        print(json.dumps(run_gemm(gemm([1], [256]), FP8, 4, 8192, [[256]])))
        """)
    assert out[0] == 0 and _kernel(out[2]) == ["SkinnyGemmStreamKernel"]
    assert (" cluster=1 " not in out[2][0]) == clusters, out[2]


@pytest.mark.parametrize("dtype,n", [("BF16", 256), ("FP8", 256), ("U8", 256), ("U8", 128)])
def test_a_stage_is_made_of_whole_boxes(fake, dtype, n):  # noqa: F811
    """A box has at most 256 rows and begins on 128 bytes.  17 warps along K make 544 rows, which three boxes are not; where rows
    are copied in pairs (NVFP4, N an odd multiple of 128) they are two boxes of 136 of either kind."""
    width = 1 if dtype == "U8" else 3
    out = fake(f"""
        print(json.dumps([run_gemm(gemm([1], [{n}], stream_plan="{width},%d,1,1" % wk), {dtype}, 1, 4096, [[{n}]]) for wk in range(1, 19)]))
        """)
    for wk, (code, message, log) in enumerate(out, 1):
        if wk == 17 and n == 256:
            assert code != 0 and "stream_plan" in message and log == []
        else:
            assert code == 0 and _kernel(log) == ["SkinnyGemmStreamKernel"], (wk, message)


@pytest.mark.parametrize("dtype", ["BF16", "FP8", "U8"])
def test_a_device_that_refuses_the_kernel(fake, dtype):  # noqa: F811
    """Its shared-memory limit could not be raised: nodes are made, and their calls are the general kernels'."""
    out = fake(f"""
        fake.fake_refuse_setup_of(b"SkinnyGemmStreamKernel")
        r = [run_gemm(gemm([1], [256]), {dtype}, 2, 512, [[256]]), run_shared(shared(), {dtype}, 3, 256, 128)]
        print(json.dumps(r + [run_gemm(gemm([1], [256], stream_plan="1,4,1,1"), {dtype}, 2, 512, [[256]])]))
        """)
    for code, message, log in out[:2]:
        assert code == 0 and _kernel(log) == ["SkinnyGemm"], message
    assert out[2][0] != 0 and out[2][2] == []  # a pinned shape of that kernel is an error


def test_a_device_that_reports_no_resident_block(fake):  # noqa: F811
    """A few more groups of 128 columns than SMs hold: the rule for that shape divides by the resident CTAs."""
    out = fake("""
        fake.fake_resident(0)
        print(json.dumps(run_gemm(gemm([1], [128 * 600]), U8, 2, 512, [[128 * 600]])))
        """)
    assert out[0] == 0 and _kernel(out[2]) == ["SkinnyGemm"], out[1]


@pytest.mark.parametrize("dtype", ["BF16", "FP8", "U8"])
@pytest.mark.parametrize("status,overlaps", [(0, True), (1, False), (2, False), (-1, False)])
def test_launches_overlap_their_predecessor_outside_captures(fake, dtype, status, overlaps):  # noqa: F811
    """Programmatic launches where the stream is known not to be captured, plain ones otherwise; `pdl_wait` asks for the former."""
    logs = fake(f"""
        fake.fake_capturing({status})
        r = [run_gemm(gemm([1], [256]), {dtype}, m, 512, [[256]])[2] for m in (4, 40)]
        r += [run_shared(shared(), {dtype}, m, 256, 128)[2] for m in (4, 40)]
        fake.fake_clear()
        assert lib.qfg_argmax_rows(BF16, P, 4, 4096, P, P, None) == 0
        h = ctypes.c_void_p()
        assert lib.qfg_dequant_create(256, 0, None, 0, None, 0, ctypes.byref(h)) == 0
        w = L.Tensor2D(P, {dtype}, 512, cols({dtype}, 256))
        assert lib.qfg_dequant_compute(h, ctypes.byref(w), (ctypes.c_void_p * 1)(P), 1, None) == 0
        r.append(fake.fake_log().decode().split("\\n")[:-1])
        print(json.dumps(r + [run_gemm(gemm([1], [256], pdl_wait=1), {dtype}, 4, 512, [[256]])[2]]))
        """)
    assert [len(log) for log in logs] == [1, 1, 1, 1, 2, 1]
    assert all(line.endswith(f"pdl={int(overlaps)}") for log in logs[:5] for line in log)
    assert logs[5][0].endswith("pdl=1")
