"""Scheduling for the B200 backend: one fused node group -> one template instantiation.

Counterpart of ``NPUTritonScheduling`` (``inductor_x/codegen/schduling.py:24-163``).  The
reference overrides ``codegen_node_schedule`` to un-flatten the indexing of every node into
true axes before picking split/tiling axes (``decide_codegen_dims_in_kernel``); here the
stock SIMD flow is kept and the un-flattening questions are answered per access by
``codegen/ir.py`` while the kernel is emitted.  Tiling is always the flat
``(numel, rnumel)`` pair, as in the reference's ``select_tiling`` patch
(``inductor_x/codegen/triton.py:175-177``).
"""
from __future__ import annotations

import copy

import sympy
import torch
from torch._inductor import config as inductor_config
from torch._inductor.codegen.common import BackendFeature
from torch._inductor.codegen.simd import SIMDScheduling
from torch._inductor.dependencies import MemoryDep
from torch._inductor.scheduler import SchedulerNode
from torch._inductor.utils import get_kernel_metadata
from torch._inductor.virtualized import V
from torch.utils._ordered_set import OrderedSet

from .. import config
from . import split_tiling
from .kernel import B200Kernel

HEADER = "from inductor_x_b200.codegen.jit import load_kernel as ixb_load_kernel"


class ColumnSumNode(SchedulerNode):
    """A sum over the rows of a matrix, emitted inside the row kernel that works on the same rows: the
    row's index takes the place of its reduced one."""

    @classmethod
    def of(cls, node: SchedulerNode, ranges, casts) -> "ColumnSumNode":
        out = copy.copy(node)
        out.__class__ = cls
        # casts: buffer of a sum -> the node that converts it, which the sum's store takes over
        out.swapped, out.casts = ranges, {b: c for b, c in casts.items() if b in node.get_buffer_names()}
        return out

    def mark_run(self) -> None:
        super().mark_run()
        for cast in self.casts.values():
            cast.mark_run()

    def get_ranges(self):
        return self.swapped

    def is_reduction(self) -> bool:
        return False

    def codegen(self, index_vars) -> None:
        rows, columns = index_vars
        V.kernel.column_mode = True
        V.kernel.column_casts = {b: next(iter(c.get_buffer_names())) for b, c in self.casts.items()}
        try:
            super().codegen((columns, rows))
        finally:
            V.kernel.column_mode = False


class ColumnGroup:
    """A group of sums over the rows of dense [rows, cols] matrices, each stored as it is or converted
    once; ``of`` gives None for any other group."""

    def __init__(self, nodes, sums, casts, matrices, rows, cols):
        self.nodes, self.sums, self.casts, self.matrices, self.rows, self.cols = nodes, sums, casts, matrices, rows, cols
        self.reads = {d.name for n in sums for d in n.read_writes.reads}
        self.writes = {name for n in nodes for name in n.get_buffer_names()}

    @classmethod
    def of(cls, group):
        nodes = group.get_nodes()
        if not all(type(n) is SchedulerNode for n in nodes):
            return None
        sums = [n for n in nodes if n.is_reduction()]
        if not sums:
            return None
        cols, rows = (_static(v) for v in sums[0].group[1])
        if cols is None or rows is None or rows < 128:
            return None
        # slow on its own, or few rows to a block of its own (see config; fp32 rows of four over a multiple of
        # eight belong here as well: 2000 x 2044 17.2 us in two kernels, 12.9 in one, 1500 x 3004 21.0 and 11.8.
        # bf16 of 4096 columns and less gains nothing below the other threshold, 512 x 6144 10.0 / 8.8,
        # 800 x 6144 13.0 / 10.6)
        odd = cols % 8 != 0 or cols >= 6144
        if rows * cols < (config.column_sum_elements_odd if odd else config.column_sum_elements):
            return None
        matrices, made = set(), {}
        for n in sums:
            data = getattr(n.node, "data", None)
            if [_static(v) for v in n.group[1]] != [cols, rows] or getattr(data, "reduction_type", None) != "sum" or \
                    data.src_dtype not in (torch.float32, torch.float16, torch.bfloat16) or \
                    [[_static(v) for v in r] for r in n.get_ranges()] != [[cols], [rows]]:
                return None
            for d in n.read_writes.reads:
                if not isinstance(d, MemoryDep) or [_static(v) for v in d.size] not in ([cols, rows], [rows], [cols]):
                    return None
                if len(d.size) == 2:
                    c, r = d.var_names
                    if sympy.expand(d.index - c - cols * r) == 0:
                        matrices.add(d.name)
                    elif {c, r} <= d.index.free_symbols:
                        return None
            made.update({name: n for name in n.get_buffer_names()})
        casts = {}
        for n in nodes:
            if n in sums:
                continue
            reads, writes = list(n.read_writes.reads), list(n.get_buffer_names())
            if getattr(n._body, "op_counts", None) != {"load": 1, "to_dtype": 1, "store": 1, "output": 1} or len(reads) != 1 or len(writes) != 1 or \
                    reads[0].name not in made or reads[0].name in casts or _dtype(reads[0].name) != torch.float32:
                return None
            users = {u.node.get_name() for out in made[reads[0].name].get_outputs() for u in out.users}
            index = reads[0].index
            if users != {n.get_name()} or [_static(v) for v in reads[0].size] != [cols] or index != reads[0].var_names[0] or \
                    [w.index for w in n.read_writes.writes] != [index]:
                return None
            casts[reads[0].name] = n
        return cls(nodes, sums, casts, matrices, rows, cols) if matrices else None

    def members(self):
        ranges = ([sympy.Integer(self.rows)], [sympy.Integer(self.cols)])
        return [ColumnSumNode.of(n, ranges, self.casts) for n in self.sums]

    def fits(self, group) -> bool:
        """``group`` is one of row reductions over the same rows, worked on by the row template, that
        reads all that the sums read (so that none of it is given back or written over before)
        and has nothing to do with their results, and its threads can hold their part of the sums."""
        if not _is_generated(group) or not group.is_reduction() or \
                [_static(v) for v in group.group[1]] != [self.rows, self.cols]:
            return False
        reads, writes = {d.name for d in _reads(group)}, set(group.get_buffer_names())
        if not self.reads <= reads or self.reads & writes or reads & self.writes:
            return False
        seen, dtypes = set(), []
        for d in _reads(group):
            if d.name not in self.matrices:
                continue
            if not isinstance(d, MemoryDep):
                return False
            # from the beginning, element after element
            stride, expected = 1, sympy.S.Zero
            for v, size in zip(reversed(d.var_names), reversed(d.size)):
                if _static(size) is None:
                    return False
                expected += v * stride
                stride *= int(size)
            if stride != self.rows * self.cols or sympy.expand(d.index - expected) != 0:
                return False
            seen.add(d.name)
        # (what the kernel will see: a conversion is not a node of it)
        for n in [*group.get_nodes(), *self.sums]:
            dtypes += [_dtype(d.name) for d in [*n.read_writes.reads, *n.read_writes.writes]]
        floats = [d for d in dtypes if d in (torch.float32, torch.float16, torch.bfloat16)]
        if None in dtypes or seen != self.matrices or len(floats) != len([d for d in dtypes if d.is_floating_point]):
            return False
        narrowest = split_tiling.narrowest_dtype(floats)
        if split_tiling.walked_in_chunks(self.cols, narrowest):
            return False          # a thread's sums are those of one chunk
        shape = split_tiling.choose_row_config(self.cols, narrowest, rows=self.rows)
        # whole warps to a row, and at most 64 registers of sums in the default launch shape
        return shape is not None and shape.team >= 32 and shape.vec % 4 == 0 and \
            shape.elems_per_thread * len(self.sums) <= 64 and self._pays(shape, narrowest)

    def _pays(self, shape, dtype) -> bool:
        """One kernel is quicker than two.  A kernel of its own reads the matrices a second time, and is
        slow where it is two sums (two passes) or where the last 32 vectors of a row are not whole (they
        are read one load at a time, and the rest waits for them).  Beside the row the sums take registers,
        of which a thread of a 1024-thread team has 64, and where there are few rows to a block its partial
        sums are as much as what they spare.  Backward of a norm, two kernels / one, us:
          one sum, whole vectors, 1024 threads: bf16 448 x 16384 17.6 / 22.9, 4096 x 16384 109 / 125,
            1024 x 24576 66 / 78, 1024 x 32768 103 / 156; fp32 700 x 16384 57.9 / 57.0, 4096 x 16384 293 / 269,
            1024 x 24576 159 / 205.  Fewer threads: bf16 1024 x 12288 23.4 / 18.7, 400 x 8192 10.7 / 8.5,
            256 x 12288 9.6 / 10.6
          one sum, ragged: bf16 220 x 16000 21.3 / 16.6, 200 x 16383 31.7 / 27.7, 1024 x 24571 173 / 101,
            256 x 32767 65 / 85, 512 x 32767 123 / 131, 2048 x 32767 509 / 463, 300 x 50257 146 / 200,
            512 x 65535 528 / 540; fp32 256 x 16383 40 / 35, 2048 x 16383 283 / 167
          two sums: bf16 400 x 16384 62 / 41, 256 x 16384 28 / 34, 1024 x 32768 339 / 323, 512 x 32767 162 / 274,
            2048 x 32767 785 / 873; fp32 1024 x 20000 251 / 198, 1024 x 16383 174 / 147
        Where the words of a row are shifted one by one (it fills its team) two sums have no registers.
        With equal thresholds the kernel of its own counts as slow everywhere."""
        full = False
        if self.cols % shape.vec:
            shifted = split_tiling.covering_config(self.cols, dtype, shape, 0, rows=self.rows)
            full, shape = shifted is None, shifted or shape
        quick = len(self.sums) == 1 and self.cols % (32 * shape.vec) == 0 and \
            config.column_sum_elements > config.column_sum_elements_odd
        few = self.rows < 400
        if shape.team < split_tiling.MAX_TEAM:
            return not (quick and few)
        elems = shape.elems_per_thread
        if quick:
            return not few and shape.vec == 4 and elems <= 16
        if few:
            return not full and elems * len(self.sums) <= 20
        if full and len(self.sums) > 1:
            return False
        return elems <= 32 or (elems <= 40 and len(self.sums) == 1 and self.rows >= 1024)

    def is_touched_by(self, group) -> bool:
        """A group between the two wants the sums, or writes what they are made of."""
        return bool({d.name for d in _reads(group)} & self.writes or set(group.get_buffer_names()) & self.reads or
                    any(self.reads & set(out.get_mutations()) for out in group.get_outputs()))


def _static(numel):
    return int(numel) if isinstance(numel, int) or getattr(numel, "is_Integer", False) else None


def _dtype(name):
    try:
        return V.graph.get_dtype(name)
    except Exception:
        return None


def _is_generated(node) -> bool:
    return type(node).__name__ in ("SchedulerNode", "FusedSchedulerNode")


def _reads(node):
    return [d for n in node.get_nodes() for d in n.read_writes.reads]


class B200Scheduling(SIMDScheduling):
    kernel_type = B200Kernel  # type: ignore[assignment]

    def __init__(self, scheduler) -> None:
        super().__init__(scheduler)
        self._put_off: dict = {}      # id of a row group -> the column sums to be emitted with it
        self._done: dict = {}         # groups of column sums that a row kernel before them has emitted
        self._beside = None
        wrapper = V.graph.wrapper_code
        if wrapper is not None:
            wrapper.header.splice(HEADER)

    @classmethod
    def get_backend_features(cls, device):
        # no tuple reductions: var_mean is lowered to the two-pass form, as the reference
        # does (inductor_x/lowering.py:270-325); scans only in the form the lowering lets
        # through (a sum along a stride-1 row held on chip); no sorts / foreach
        return OrderedSet([BackendFeature.INPLACE_BUFFERS, BackendFeature.REDUCE_TO_SINGLE_ELEMENT,
                           BackendFeature.SCAN])

    @classmethod
    def get_tiling_and_scores(cls, node_schedule, numel, reduction_numel=sympy.S.One,
                              coalesce_analysis=None):
        # always the flat (numel, rnumel) pair; pointwise groups carry rnumel == 1, which is
        # also what lets the scheduler fuse them into a reduction of the same rows
        return {"x": numel, "r0_": reduction_numel}, None

    @classmethod
    def select_tiling(cls, node_schedule, numel, reduction_numel=sympy.S.One, coalesce_analysis=None):
        return cls.get_tiling_and_scores(node_schedule, numel, reduction_numel)[0]

    # ---- sums over the rows beside a row kernel ------------------------------------------------
    # The backward of a norm reads the same matrices twice: row by row for the gradient of its input,
    # column by column for those of its weight and bias (sum over the tokens of dy * x * rstd).  Where
    # the two groups come close enough after each other the sums are emitted inside the row kernel
    # (gen.cuh, finish_columns), in its turn: the one that comes first waits for the other, or the
    # other is found done.  32768 x 4096 bf16: 121 + 88 us in two kernels, 123 + 4 in one.
    # How many groups after the first the second may come.  In the backward of encoder and decoder layers it
    # is the next one; the bound keeps the search short in graphs of thousands.
    COLUMN_SUM_WINDOW = 8

    def codegen_node(self, node):
        if self._done.pop(id(node), None) is not None:
            return None
        # (combo kernels are emitted past this function)
        if config.merged_column_sums and not inductor_config.combo_kernels and id(node) not in self._put_off:
            sums = ColumnGroup.of(node)
            partner = self._partner(node, sums.fits, sums) if sums else None
            if partner is not None:
                self._put_off[id(partner)] = sums
                return None
            found = {}

            def goes_beside(later):
                group = ColumnGroup.of(later)
                if group is None or not group.fits(node):
                    return False
                found["sums"] = group
                return True

            later = self._partner(node, goes_beside) if node.is_reduction() else None
            if later is not None and not any(found["sums"].is_touched_by(n) for n in self._between(node, later)):
                self._done[id(later)] = later
                self._put_off[id(node)] = found["sums"]
        self._beside = self._put_off.pop(id(node), None)
        try:
            return super().codegen_node(node)
        finally:
            self._beside = None

    def generate_node_schedule(self, nodes, numel, rnumel):
        schedule = super().generate_node_schedule(nodes, numel, rnumel)
        if self._beside is not None:
            # ahead of the rest: its operands are read before the row may be overwritten in place
            schedule = self._beside.members() + list(schedule)
        return schedule

    def _between(self, node, later):
        order = self.scheduler.nodes
        at = next(i for i, n in enumerate(order) if n is node)
        to = next(i for i, n in enumerate(order) if n is later)
        return order[at + 1:to]

    def _partner(self, node, wanted, sums=None):
        """The first group after ``node``, within the window, that is ``wanted`` and is in no pair yet;
        with ``sums`` the search ends at a group that they must not wait for."""
        order = self.scheduler.nodes
        at = next((i for i, n in enumerate(order) if n is node), None)
        if at is None:
            return None
        for later in order[at + 1:at + 1 + self.COLUMN_SUM_WINDOW]:
            if _is_generated(later) and id(later) not in self._put_off and \
                    id(later) not in self._done and later.get_device() == node.get_device() and wanted(later):
                return later
            if inductor_config.graph_partition and not (_is_generated(later) and later.get_device() == node.get_device()):
                return None      # what follows may belong to another partition of the graph
            if sums is not None and sums.is_touched_by(later):
                return None
        return None

    def define_kernel(self, src_code, node_schedule, kernel) -> str:
        wrapper = V.graph.wrapper_code
        if src_code in wrapper.src_to_kernel:
            return wrapper.src_to_kernel[src_code]
        family = getattr(kernel, "mapping", "row" if kernel.is_row else "pointwise")
        kernel_name = f"ixb_{family}_{wrapper.next_kernel_suffix()}"
        wrapper.src_to_kernel[src_code] = kernel_name
        origins, detailed = get_kernel_metadata(node_schedule, wrapper)
        wrapper.define_kernel(kernel_name, src_code, f"{origins}\n{detailed}", gpu=False)
        return kernel_name

    def codegen_sync(self) -> None:
        V.graph.wrapper_code.writeline(V.graph.device_ops.synchronize())

    def can_fuse_multi_outputs_template(self, node1, node2) -> bool:
        return False
