"""Command calls on host storage around the sizes where their paths change: element groups against padded channel tails and
bank-line padding, folds of a few long chains, storage read in place (up to 1 MiB) against storage copied in pieces."""
import time

import numpy as np
import pytest
import torch

from vibe_compiler_b200 import _abi as abi
from vibe_compiler_b200.backend import B200TargetModelBackend, FormalGemmOperation, NumericTensor, PhysicalTensorDescriptor, WB200Error
from vibe_compiler_b200.tile_program import TileProgram

pytestmark = pytest.mark.gpu
LAYOUTS = {"tensor": abi.LAYOUT_TENSOR, "cx": abi.LAYOUT_CX, "ncx": abi.LAYOUT_NCX}


def physical(backend, key, values):
    """Storage holding `values` (uint bit patterns, row-major), 0x5a in every padding byte."""
    blank = np.full(B200TargetModelBackend.physical_bytes(key), 0x5a, dtype=np.uint8)
    return backend.pack(key, values, blank)


def logical(backend, key, storage, dtype):
    return backend.unpack(NumericTensor(key, storage)).view(dtype)


@pytest.mark.parametrize("layout,shape", [("tensor", [7]), ("tensor", [1003]), ("cx", [3, 5]), ("cx", [5, 66]), ("cx", [7, 97]), ("cx", [33, 64]),
                                          ("ncx", [2, 3, 65]), ("ncx", [3, 2, 5, 129]), ("ncx", [2049, 1, 64]), ("ncx", [300, 2, 97]), ("cx", [1031, 263]), ("tensor", [700001])])
def test_elementwise_and_convert_keep_padding_and_match_numpy(backend, layout, shape):
    rng = np.random.default_rng(sum(shape))
    count = int(np.prod(shape))
    x, y = (rng.standard_normal(count).astype(np.float32) for _ in range(2))
    f32, bf16 = (PhysicalTensorDescriptor(f, LAYOUTS[layout], shape) for f in (abi.F32, abi.BF16))
    blank = np.full(B200TargetModelBackend.physical_bytes(f32), 0x11, dtype=np.uint8)
    got = backend.execute_elementwise("sub", [NumericTensor(f32, physical(backend, f32, v)) for v in (x, y)], NumericTensor(f32, blank))
    assert np.array_equal(logical(backend, f32, got.destination.storage, np.float32), x - y)
    # every byte that is no element keeps the template's value
    marked = backend.pack(f32, np.full(count, 0x22222222, np.uint32), np.full_like(blank, 0x11))
    assert np.array_equal(got.destination.storage[marked == 0x11], blank[marked == 0x11])
    half = backend.execute_convert(167, got.destination, NumericTensor(bf16, np.zeros(B200TargetModelBackend.physical_bytes(bf16), np.uint8)))
    want = torch.from_numpy(x - y).bfloat16().view(torch.int16).numpy().view(np.uint16)
    assert np.array_equal(logical(backend, bf16, half.destination.storage, np.uint16), want)


@pytest.mark.parametrize("shape,dimension,axes", [([5], "trailing0", (0,)), ([65, 7], "trailing1", (0,)), ([300, 70], "trailing1", (0,)), ([3, 130], "trailing0", (1,)),
                                                  ([2, 4, 66, 65], "trailing1", (2,)), ([2, 3, 5, 97], "trailing2and1", (1, 2)),
                                                  ([2, 3, 5, 97], "trailing2and1and0", (1, 2, 3)), ([3, 2, 2, 64], "trailing3", (0,)), ([1, 1, 64, 64], "trailing1", (2,))])
@pytest.mark.parametrize("formal", [False, True])
def test_folds_follow_the_input_order(backend, shape, dimension, axes, formal):
    rng = np.random.default_rng(3)
    x = (rng.standard_normal(shape) * 10.0 ** rng.integers(-3, 4, shape)).astype(np.float32)
    x.reshape(-1)[::7] = 0.0
    x.reshape(-1)[3::11] = -0.0
    out_shape = [1 if d in axes else n for d, n in enumerate(shape)]
    chains = np.moveaxis(x, axes, tuple(range(len(axes)))).reshape(-1, int(np.prod(out_shape)))   # row-major input order per output
    for layout in (abi.LAYOUT_NCX, abi.LAYOUT_TENSOR):
        key, out_key = PhysicalTensorDescriptor(abi.F32, layout, shape), PhysicalTensorDescriptor(abi.F32, layout, out_shape)
        source = NumericTensor(key, physical(backend, key, x.reshape(-1)))
        blank = NumericTensor(out_key, np.zeros(B200TargetModelBackend.physical_bytes(out_key), np.uint8))
        total = np.zeros(chains.shape[1], np.float32)
        for row in chains:
            total = (total + row).astype(np.float32)
        got = backend.execute_reduce("sum", dimension, source, blank, formal=formal)
        assert np.array_equal(logical(backend, out_key, got.destination.storage, np.uint32), total.view(np.uint32))
        if formal:   # a step that rounds raises inexact (16); one step from +0 never does
            assert got.evidence.flags == (16 if chains.shape[0] > 1 else 0)
            whole = NumericTensor(key, physical(backend, key, np.rint(x).reshape(-1)))   # integers far below 2^24: every step is exact
            assert backend.execute_reduce("sum", dimension, whole, blank, formal=True).evidence.flags == 0
        for name, pick in (("max", chains.max(0)), ("min", chains.min(0))):
            got = backend.execute_reduce(name, dimension, source, blank, formal=formal)
            assert np.array_equal(logical(backend, out_key, got.destination.storage, np.float32), pick)
            assert got.evidence.flags == 0


def test_folds_meet_exceptional_values_inside_a_chunk(backend):
    key, out_key = PhysicalTensorDescriptor(abi.F32, abi.LAYOUT_TENSOR, [130, 3]), PhysicalTensorDescriptor(abi.F32, abi.LAYOUT_TENSOR, [1, 3])
    blank = NumericTensor(out_key, np.zeros(12, np.uint8))
    x = np.ones((130, 3), np.float32)
    x[70, 1], x[100, 2] = np.inf, np.float32(3.4e38)
    x[101, 2] = np.float32(3.4e38)                       # overflows in the middle of a chunk
    got = backend.execute_reduce("sum", "trailing1", NumericTensor(key, x), blank, formal=True)
    assert np.array_equal(got.destination.storage.view(np.float32), np.array([130, np.inf, np.inf], np.float32)) and got.evidence.flags & 4
    x[:, 0] = -0.0
    for name, want in (("max", 0x80000000), ("min", 0x80000000)):
        got = backend.execute_reduce(name, "trailing1", NumericTensor(key, x), blank, formal=True)
        assert got.destination.storage.view(np.uint32)[0] == want
    x[66, 0] = np.nan
    got = backend.execute_reduce("max", "trailing1", NumericTensor(key, x), blank, formal=True)
    assert got.destination.storage.view(np.uint32)[0] == 0x7fc00000
    with pytest.raises(WB200Error):
        backend.execute_reduce("max", "trailing1", NumericTensor(key, x), blank)


@pytest.mark.parametrize("elements", [(1 << 18) - 1, 1 << 18, (1 << 18) + 1, (9 << 20) + 5])
def test_storage_in_place_and_in_pieces(backend, elements):
    rng = np.random.default_rng(elements)
    x, y = (rng.standard_normal(elements).astype(np.float32) for _ in range(2))
    key = PhysicalTensorDescriptor(abi.F32, abi.LAYOUT_TENSOR, [elements])
    got = backend.execute_elementwise("add", [NumericTensor(key, x), NumericTensor(key, y)], NumericTensor(key, np.zeros(4 * elements, np.uint8)))
    assert np.array_equal(got.destination.storage.view(np.float32), x + y)


MIB = 1 << 20


# operands of as many bytes as the 32 MiB transfer area holds, once and one and a half times over
@pytest.mark.parametrize("each", [16 * MIB, 24 * MIB])
def test_flags_are_read_back_behind_operands_that_fill_the_transfer_area(backend, each):
    key = PhysicalTensorDescriptor(abi.F32, abi.LAYOUT_TENSOR, [each // 4])
    x = np.arange(each // 4, dtype=np.float32)
    got = backend.execute_elementwise("add", [NumericTensor(key, x), NumericTensor(key, x)], NumericTensor(key, np.zeros(each, np.uint8)), formal=True)
    assert np.array_equal(got.destination.storage.view(np.float32), x + x) and got.evidence.flags == 0
    key, out_key = (PhysicalTensorDescriptor(abi.F32, abi.LAYOUT_TENSOR, [rows, each // 128]) for rows in (64, 1))
    x = np.arange(each // 2, dtype=np.float32) % 127
    got = backend.execute_reduce("sum", "trailing1", NumericTensor(key, x), NumericTensor(out_key, np.zeros(each // 32, np.uint8)), formal=True)
    assert np.array_equal(got.destination.storage.view(np.float32), x.reshape(64, -1).sum(0)) and got.evidence.flags == 0   # small integers: exact


def test_program_with_inputs_that_fill_the_transfer_area(backend):
    count = 32   # of 1 MiB, the largest that go through the area
    rows = [f'!{{i64 {i}, !"external-input", i64 {i}, !"", !"f32", !"tensor", i64 {MIB}, i64 {MIB // 4}, !"read-only", i64 {MIB // 256}, i64 64, i64 0}}'
            for i in range(count)]
    rows.append(f'!{{i64 {count}, !"external-output", i64 0, !"", !"f32", !"tensor", i64 1024, i64 256, !"write-only", i64 4, i64 64, i64 0}}')
    lines = [f"define void @entry({', '.join(f'i64 %{i}' for i in range(count + 1))}) {{", f"  %src = add i64 %{count - 1}, {MIB - 1024}",
             "  call void @wafer_tx81_rdma(i64 %src, i64 0, i32 1024, i32 1024, i32 0, i32 0, i32 0, i32 1, i32 1, i32 1, i32 5, i32 0)",
             f"  call void @wafer_tx81_wdma(i64 0, i64 %{count}, i32 1024, i32 1024, i32 0, i32 0, i32 0, i32 1, i32 1, i32 1, i32 5, i32 0)",
             "  ret void", "}", "!wafer.target.tile_id = !{!2}",
             f"!wafer.target.entry_arguments = !{{{', '.join(f'!{10 + i}' for i in range(count + 1))}}}", "!2 = !{i64 0}"]
    module = "\n".join(lines + [f"!{10 + i} = {row}" for i, row in enumerate(rows)]) + "\n"
    x = np.arange(count * MIB // 4, dtype=np.float32).reshape(count, -1, 64)
    (out,), _ = TileProgram([module], backend, spm_bytes=1 << 16).run(list(x))
    assert np.array_equal(out.view(np.float32).reshape(-1), x.reshape(-1)[-256:])


def pinned(data):
    """A page-locked copy of `data`'s bytes."""
    return torch.from_numpy(data.view(np.uint8).reshape(-1)).pin_memory().numpy()


def into(monkeypatch, storage):
    """Makes the next command write its result to `storage`, as a C caller may name any destination."""
    monkeypatch.setattr(B200TargetModelBackend._results, "empty", lambda size: storage[:size])


# Results over their own page-locked operands, in layouts whose padding comes from the template: the operands are read first.
def test_padded_result_over_a_page_locked_operand(backend, monkeypatch):
    rng = np.random.default_rng(5)
    square = PhysicalTensorDescriptor(abi.F32, abi.LAYOUT_CX, [321, 321])
    lhs, rhs = (physical(backend, square, rng.standard_normal(321 * 321).astype(np.float32).view(np.uint32)) for _ in range(2))
    blank = NumericTensor(square, np.full(B200TargetModelBackend.physical_bytes(square), 0x11, np.uint8))
    operation = FormalGemmOperation(square, square, square, 321, 321, 321)
    halves = [PhysicalTensorDescriptor(f, abi.LAYOUT_CX, [300, 97]) for f in (abi.BF16, abi.F16)]
    source = physical(backend, halves[0], rng.integers(0x3f00, 0x4100, 300 * 97).astype(np.uint16))
    spare = NumericTensor(halves[1], np.full(B200TargetModelBackend.physical_bytes(halves[1]), 0x11, np.uint8))

    def commands(lhs, rhs, source):
        yield lhs, lambda: backend.try_execute(operation, NumericTensor(square, lhs), NumericTensor(square, rhs), blank, policy=abi.GEMM_FORMAL)
        yield rhs, lambda: backend.try_execute(operation, NumericTensor(square, lhs), NumericTensor(square, rhs), blank, policy=abi.GEMM_FORMAL)
        yield source, lambda: backend.execute_convert(154, NumericTensor(halves[0], source), spare, formal=True)
    for index in range(3):
        want = list(commands(lhs, rhs, source))[index][1]().destination.storage.copy()
        with monkeypatch.context() as patch:
            over, command = list(commands(pinned(lhs), pinned(rhs), pinned(source)))[index]
            into(patch, over)
            assert np.array_equal(command().destination.storage, want)


@pytest.mark.parametrize("start", [0, 1 << 17])
def test_storage_of_which_only_a_part_is_registered(backend, start):
    elements = 1 << 16
    room = np.zeros(4 * elements + 4096, np.uint8)
    lead = -room.ctypes.data % 4096
    x = room[lead:lead + 4 * elements].view(np.float32)
    x[:] = np.arange(elements)
    runtime = torch.cuda.cudart()
    assert runtime.cudaHostRegister(x.ctypes.data + start, 1 << 17, 0) == runtime.cudaError.success   # half of the operand
    try:
        key = PhysicalTensorDescriptor(abi.F32, abi.LAYOUT_TENSOR, [elements])
        got = backend.execute_elementwise("add", [NumericTensor(key, x), NumericTensor(key, x)], NumericTensor(key, np.zeros(4 * elements, np.uint8)))
        assert np.array_equal(got.destination.storage.view(np.float32), x + x)
    finally:
        runtime.cudaHostUnregister(x.ctypes.data + start)


def test_ragged_product_under_the_tensor_policy_reads_its_operands_on_the_device(backend):
    """A product the tensor-core kernel does not take runs on the bit-exact kernel, which reads operands many times: the same bits,
    in about the time of the bit-exact policy (read over PCIe instead, this one took six times as long)."""
    m, k, n = 4001, 1005, 4003
    lhs_key, rhs_key, out_key = (PhysicalTensorDescriptor(abi.BF16, abi.LAYOUT_CX, shape) for shape in ([m, k], [k, n], [m, n]))
    rng = np.random.default_rng(2)
    lhs, rhs = (NumericTensor(key, pinned(physical(backend, key, rng.integers(0x3e00, 0x4000, key.element_count).astype(np.uint16)))) for key in (lhs_key, rhs_key))
    blank = NumericTensor(out_key, np.zeros(B200TargetModelBackend.physical_bytes(out_key), np.uint8))
    operation = FormalGemmOperation(lhs_key, rhs_key, out_key, m, k, n)
    best, results = {}, {}
    for policy in (abi.GEMM_FORMAL, abi.GEMM_TENSOR) * 4:
        begin = time.perf_counter()
        results[policy] = backend.try_execute(operation, lhs, rhs, blank, policy=policy).destination.storage
        best[policy] = min(best.get(policy, 1e9), time.perf_counter() - begin)
    assert np.array_equal(results[abi.GEMM_FORMAL], results[abi.GEMM_TENSOR])
    assert best[abi.GEMM_TENSOR] < 2 * best[abi.GEMM_FORMAL], best


@pytest.mark.parametrize("m,n", [(33, 17), (256, 321), (700, 1001), (2049, 1003)])   # results staged, page-locked, in pieces
def test_bit_exact_product_returns_through_every_kind_of_result_storage(backend, monkeypatch, m, n):
    """The same bits and the template's padding, whether the result's storage is page-locked or pageable, apart from the template or
    the template itself."""
    k = 65
    lhs_key, rhs_key, out_key = (PhysicalTensorDescriptor(abi.BF16, abi.LAYOUT_CX, shape) for shape in ([m, k], [k, n], [m, n]))
    rng = np.random.default_rng(m)
    a, b = (rng.integers(-8, 9, shape).astype(np.float32) for shape in ((m, k), (k, n)))   # small integers: every sum is exact
    half = lambda x: torch.from_numpy(x.reshape(-1)).bfloat16().view(torch.int16).numpy().view(np.uint16)
    lhs, rhs = NumericTensor(lhs_key, physical(backend, lhs_key, half(a))), NumericTensor(rhs_key, physical(backend, rhs_key, half(b)))
    operation = FormalGemmOperation(lhs_key, rhs_key, out_key, m, k, n)
    size = B200TargetModelBackend.physical_bytes(out_key)
    want = backend.pack(out_key, half(a @ b), np.full(size, 0x33, np.uint8))
    for storage in (pinned(np.zeros(size, np.uint8)), np.zeros(size, np.uint8)):
        for template in (np.full(size, 0x33, np.uint8), storage):
            storage[:] = 0x33
            with monkeypatch.context() as patch:
                into(patch, storage)
                got = backend.try_execute(operation, lhs, rhs, NumericTensor(out_key, template), policy=abi.GEMM_FORMAL)
            assert np.array_equal(got.destination.storage, want)


def scattered_commands(backend):
    """Commands whose kernels store one element at a time, with a result of 4 MB: name -> (descriptor, command)."""
    key, other = (PhysicalTensorDescriptor(f, abi.LAYOUT_CX, [2000, 1030]) for f in (abi.BF16, abi.F16))
    blank, other_blank = (NumericTensor(k, np.zeros(B200TargetModelBackend.physical_bytes(k), np.uint8)) for k in (key, other))
    thin, wide = (PhysicalTensorDescriptor(abi.BF16, abi.LAYOUT_CX, shape) for shape in ([2000, 64], [64, 1030]))
    lhs, rhs = (NumericTensor(k, np.zeros(B200TargetModelBackend.physical_bytes(k), np.uint8)) for k in (thin, wide))
    product = FormalGemmOperation(thin, wide, key, 2000, 64, 1030)
    return {"gemm": (key, lambda: backend.try_execute(product, lhs, rhs, blank, policy=abi.GEMM_FORMAL)),
            "add": (key, lambda: backend.execute_elementwise("add", [blank, blank], blank, formal=True)),
            "convert": (other, lambda: backend.execute_convert(154, blank, other_blank, formal=True))}


@pytest.mark.parametrize("name", ["gemm", "add", "convert"])
def test_page_locked_results_of_element_wise_stores_are_not_slower(backend, monkeypatch, name):
    """A large result goes through device memory and one copy whatever its storage (stored over PCIe it took three times as long
    with page-locked storage as with pageable storage)."""
    key, command = scattered_commands(backend)[name]
    size, best = B200TargetModelBackend.physical_bytes(key), {}
    for _ in range(4):
        for kind, storage in (("pageable", np.zeros(size, np.uint8)), ("page-locked", pinned(np.zeros(size, np.uint8)))):
            with monkeypatch.context() as patch:
                into(patch, storage)
                begin = time.perf_counter()
                command()
                best[kind] = min(best.get(kind, 1e9), time.perf_counter() - begin)
    assert best["page-locked"] < 1.5 * best["pageable"], best


@pytest.mark.parametrize("shape,layout", [([512, 5], "cx"), ([300, 97], "cx"), ([30000], "tensor")])
def test_refused_formal_convert_leaves_page_locked_storage(backend, monkeypatch, shape, layout):
    key, out_key = (PhysicalTensorDescriptor(f, LAYOUTS[layout], shape) for f in (abi.F32, abi.I32))
    values = np.ones(key.element_count, np.float32)
    values[7] = np.inf
    storage = pinned(np.full(B200TargetModelBackend.physical_bytes(out_key), 0x77, np.uint8))
    source, template = NumericTensor(key, physical(backend, key, values)), NumericTensor(out_key, np.zeros(storage.size, np.uint8))
    opcode = 165   # F32 -> I32
    into(monkeypatch, storage)
    with pytest.raises(WB200Error, match="float-to-integer-non-finite"):
        backend.execute_convert(opcode, source, template, formal=True)
    assert (storage == 0x77).all()
    values[7] = 3
    got = backend.execute_convert(opcode, NumericTensor(key, physical(backend, key, values)), template, formal=True)
    assert np.array_equal(logical(backend, out_key, got.destination.storage, np.int32), values.astype(np.int32))


def test_refused_program_leaves_page_locked_outputs(backend, monkeypatch):
    rows = [f'!{{i64 {i}, !"external-{kind}", i64 0, !"", !"{form}", !"tensor", i64 32768, i64 8192, !"{access}-only", i64 128, i64 64, i64 0}}'
            for i, (kind, form, access) in enumerate((("input", "f32", "read"), ("output", "i32", "write")))]
    module = f"""define void @entry(i64 %0, i64 %1) {{
  call void @wafer_tx81_rdma(i64 %0, i64 0, i32 32768, i32 32768, i32 0, i32 0, i32 0, i32 1, i32 1, i32 1, i32 5, i32 0)
  call void @wafer_tx81_convert_fp32_int32(i64 0, i64 32768, i32 8192, i32 0, i32 0, i32 1)
  call void @wafer_tx81_wdma(i64 32768, i64 %1, i32 32768, i32 32768, i32 0, i32 0, i32 0, i32 1, i32 1, i32 1, i32 4, i32 0)
  ret void
}}
!wafer.target.tile_id = !{{!2}}
!wafer.target.entry_arguments = !{{!10, !11}}
!2 = !{{i64 0}}
!10 = {rows[0]}
!11 = {rows[1]}
"""
    program = TileProgram([module], backend, spm_bytes=1 << 17)
    values = np.arange(8192, dtype=np.float32).reshape(128, 64)
    storage = pinned(np.full(32768, 0x77, np.uint8))
    into(monkeypatch, storage)
    for _ in range(2):   # the second run relaunches the graph
        values[3, 1] = np.nan
        storage[:] = 0x77
        with pytest.raises(WB200Error, match="float-to-integer-non-finite"):
            program.run([values])
        assert (storage == 0x77).all()
        values[3, 1] = 5.0
        (out,), _ = program.run([values])
        assert np.array_equal(out.view(np.int32), values.astype(np.int32))


def test_padded_result_over_a_page_locked_operand_that_is_not_aligned(backend, monkeypatch):
    """Such an operand is copied, asynchronously beyond 1 MiB, and its storage counts as an operand's all the same."""
    key, out_key = (PhysicalTensorDescriptor(f, abi.LAYOUT_CX, [1500, 1030]) for f in (abi.F32, abi.BF16))
    size, out_size = (B200TargetModelBackend.physical_bytes(k) for k in (key, out_key))
    source = physical(backend, key, np.random.default_rng(4).standard_normal(key.element_count).astype(np.float32).view(np.uint32))
    blank = NumericTensor(out_key, np.full(out_size, 0x11, np.uint8))
    want = backend.execute_convert(167, NumericTensor(key, source), blank).destination.storage.copy()
    room = pinned(np.zeros(size + 4096, np.uint8))
    room[8:8 + size] = source
    into(monkeypatch, room)   # the result begins 8 bytes before the operand
    got = backend.execute_convert(167, NumericTensor(key, room[8:8 + size]), blank)
    assert np.array_equal(got.destination.storage, want)
