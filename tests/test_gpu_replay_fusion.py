"""Which commands of one Tile a replay fuses, by the kernels it launches, and that the scratch-pad and DDR end as the CPU replay
of the commands one by one leaves them: DMA commands and elementwise commands that depend on one another in every way."""
import numpy as np
import pytest

from vibe_compiler_b200.tile_program import TileProgram

_SPM = 16384    # bytes of the scratch-pad that the programs use, loaded first and stored last
_WORK = 8192    # bytes of DDR behind the stored scratch-pad, for the DMA commands under test
_CALL = "  call void @wafer_tx81_"
_FLAT = "i32 {0}, i32 {0}, i32 0, i32 0, i32 0, i32 1, i32 1, i32 1, i32 8, i32 0"


def _module(body):
    body = "\n".join([f"{_CALL}rdma(i64 %0, i64 0, {_FLAT.format(_SPM)})", f"{_CALL}ncc_join(i32 1)", *body, f"{_CALL}ncc_join(i32 1)",
                      f"{_CALL}wdma(i64 0, i64 %1, {_FLAT.format(_SPM)})"])
    rows = [f'!{{i64 {i}, !"external-{kind}", i64 0, !"", !"u8", !"tensor", i64 {size}, i64 {size}, !"{access}-only", i64 {size}, i64 0}}'
            for i, (kind, size, access) in enumerate((("input", _SPM, "read"), ("output", _SPM + _WORK, "write")))]
    return (f"define void @entry(i64 %0, i64 %1) {{\n  %work = add i64 %1, {_SPM}\n{body}\n  ret void\n}}\n!wafer.target.tile_id = !{{!2}}\n"
            "!wafer.target.entry_arguments = !{!10, !11}\n!2 = !{i64 0}\n" + "\n".join(f"!{10 + i} = {row}" for i, row in enumerate(rows)) + "\n")


def _check(backend, module, data, launches):
    from oracle import binding, trace_replay
    binding.build()
    program = TileProgram([module], backend, spm_bytes=1 << 16)
    commands, _ = program.trace()
    source, target = program.placement(False, 0), program.placement(True, 0)
    for _ in range(2):   # the first run captures, the second relaunches; DDR keeps what the first one stored
        ddr = np.zeros(source["ddr_bytes"], dtype=np.uint8)
        ddr[source["address"] - source["ddr_base"]:][:_SPM] = data
        report = {}
        trace_replay.replay(commands, ddr, 1, spm_bytes=1 << 16, report=report)
        before = backend.launch_count
        (out,), stats = program.run([data])
        assert np.array_equal(out.reshape(-1), ddr[target["address"] - target["ddr_base"]:][:_SPM + _WORK])
        assert stats["numeric_flags"] == report["numeric_flags"]
        assert backend.launch_count - before == launches + 2   # the first load and the last store


def _load(ddr, spm, size):
    return [f"  %l{ddr}_{spm} = add i64 %0, {ddr}", f"{_CALL}rdma(i64 %l{ddr}_{spm}, i64 {spm}, {_FLAT.format(size)})"]


def _load_work(at, spm, size):
    return [f"  %w{at}_{spm} = add i64 %work, {at}", f"{_CALL}rdma(i64 %w{at}_{spm}, i64 {spm}, {_FLAT.format(size)})"]


def _store(spm, at, size):
    return [f"  %s{at}_{spm} = add i64 %work, {at}", f"{_CALL}wdma(i64 {spm}, i64 %s{at}_{spm}, {_FLAT.format(size)})"]


@pytest.mark.gpu
@pytest.mark.parametrize("body,launches", [
    ([_load(4096 + 256 * i, 1024 * i, 256) for i in range(5)], 2),                     # four to a launch
    ([_load(4096, 0, 1024), _load(8192, 512, 1024)], 2),                               # load over load
    ([_load(4096, 0, 1024), _load(4608, 1024, 1024)], 1),                              # one source of two loads
    ([_store(0, 0, 1024), _store(4096, 1008, 1024)], 2),                               # store over store
    ([_store(0, 0, 1024), _store(4096, 1024, 1024), _store(512, 2048, 16)], 1),
    ([_store(0, 0, 1024), _load_work(0, 4096, 1024)], 2),                              # a load of what was stored
    ([_load(4096, 0, 1024), _store(0, 0, 1024)], 2),                                   # a store of what was loaded
    ([_store(0, 0, 1024), _load(4096, 0, 1024)], 2),                                   # a load over what is being stored
    ([_load(4096, 0, 1024), _load(8196, 2048, 1024), _load(9001, 4097, 1003)], 3),     # units of 16, 4 and 1 bytes
    ([_load(4096, 0, 1024), _load(8196, 2048, 1024), _load(9004, 4100, 1004), _load(12000, 8192, 160)], 3),
])
def test_dma_commands(backend, body, launches):
    data = np.random.default_rng(launches).integers(0, 256, _SPM, dtype=np.uint8)
    _check(backend, _module([line for part in body for line in part]), data, launches)


def _chain(count, fmt, width, *commands):
    """Commands (operation, first operand, second, destination) over vectors at multiples of 1024 bytes; an operand is a place or a
    (place, elements off it) pair, a second one also None (unary), a float bit pattern in a list, or (place, off, unit elements)."""
    at = lambda o: 1024 * o if isinstance(o, int) else 1024 * o[0] + width * o[1]
    lines = []
    for op, lhs, rhs, dst in commands:
        if rhs is None:
            lines.append(f"{_CALL}elementwise_{op}(i64 {at(lhs)}, i64 {at(dst)}, i32 {count}, i32 {fmt}, i32 1)")
        else:
            second, unit, scalar = (rhs[0], 0, 1) if isinstance(rhs, list) else (at(rhs), rhs[2] if isinstance(rhs, tuple) and len(rhs) > 2 else 0, 0)
            lines.append(f"{_CALL}elementwise_{op}(i64 {at(lhs)}, i64 {second}, i64 {at(dst)}, i32 {count}, i32 {fmt}, i32 {unit}, i32 {scalar}, i32 0, i32 1)")
    return lines


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,width", [(5, 4), (3, 2)])
@pytest.mark.parametrize("commands,launches", [
    ([("mul", 0, 1, 2), ("add", 2, 3, 4)], 1),                                    # the previous result
    ([("mul", 0, 1, 2), ("exp", 3, None, 4), ("sub", 0, 4, 5)], 1),               # first operands of their own, an earlier result second
    ([("mul", 0, 1, 2), ("add", 2, 3, 0), ("max", 0, 1, 1)], 1),                  # over earlier first and second operands
    ([("mul", 0, 1, 2), ("add", 3, 4, 2), ("sub", 2, [0x3f80], 5)], 1),           # over an earlier result
    ([("sub", 0, (8, 0, 16), 2), ("mul", 2, (8, 8, 7), 3)], 1),                   # repeated units
    ([("sub", 0, (8, 0, 16), 2), ("add", 1, 2, 8)], 2),                           # over an earlier unit
    ([("mul", 0, 1, 2), ("sub", 3, (2, 0, 16), 4)], 2),                           # a unit of an earlier result
    ([("mul", 0, 1, 2), ("sub", 3, (2, 0, 1), 4)], 2),
    ([("mul", 0, 1, 2), ("add", 3, 4, (2, 1))], 2),                               # a shifted destination
    ([("mul", 0, 1, 2), ("add", (2, 1), 3, 4)], 2),                               # shifted operands
    ([("mul", 0, 1, 2), ("add", 3, (2, 2), 4)], 2),
    ([("mul", 0, (1, 1), 2), ("add", 2, 3, 1)], 2),
    ([("sub", 0, (8, 0, 61), 2), ("add", 2, (9, 0, 64), 3)], 1),                  # units as long as the vector and longer
    ([("add", 0, 1, 2)] + [("mul", 2, [0x3f00], 2)] * 8, 2),                      # eight commands to a launch; the ninth alone
])
def test_elementwise_commands(backend, commands, launches, fmt, width):
    values = np.random.default_rng(len(commands)).uniform(-2, 2, _SPM // 4).astype(np.float32)
    data = values.view(np.uint8) if fmt == 5 else (np.repeat(values, 2).view(np.uint32) >> 16).astype(np.uint16).view(np.uint8)
    _check(backend, _module(_chain(61, fmt, width, *commands)), data, launches)


@pytest.mark.gpu
def test_commands_of_other_lengths_and_formats_stay_apart(backend):
    data = np.random.default_rng(0).uniform(-2, 2, _SPM // 4).astype(np.float32).view(np.uint8)
    body = _chain(61, 5, 4, ("mul", 0, 1, 2)) + _chain(60, 5, 4, ("mul", 2, 1, 3)) + _chain(60, 3, 2, ("mul", 3, 1, 4))
    _check(backend, _module(body), data, 3)
