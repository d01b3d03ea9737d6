"""The order in which the keep-all executors issue a step on the GPU, worked out once per feed shape.

Nine things are taken out of the node-by-node loop.  They change no value, but for the rounding of a loss whose labels
come from class ids (the same sum, added up in another order):

* element-wise operators over the same elements are collected and run as one ``tsb_pointwise`` program, at the first
  node that needs one of their results; results that nobody outside the program reads are not stored;
* a reshape of a row-major array is a view of it, and so is a slice that only products read;
* the small parameter gradients that a normalisation operator hands out from its own buffers are copied in one launch;
* small matrix products that are ready together run as one launch, and so do column sums of a few rows, which wait until
  there is a launch of them or nothing else is left to do;
* the bias of a product, and the ReLU behind it, are added where the product stores its outputs;
* one-hot labels, scaled and shifted (label smoothing), that only a cross-entropy reads are not made: it takes the ids;
* a loss and its gradient come from one pass over the logits, when the gradient is due;
* a residual addition and its ReLU are taken by the batch norm before them, where nothing else reads that;
* of two convolutions' gradients that only their sum reads, the first is written where the sum goes, and the other, if its
  stride is 2, adds itself to it.

Element-wise nodes are taken as soon as their inputs are there, the others in creation order, and nothing moves past a
node with effects of its own (an optimizer update, a collective, a swap).  The memory-planning executors have
schedules of their own and do not use this.
"""
from __future__ import annotations

import heapq

import numpy as np

from .. import ndarray
from ..ops import _gpu as G
from ..ops.conv import Conv2dGradDataOp
from ..ops.elementwise import AddConstOp, AddOp, AddReluOp, MulConstOp, ReluOp, _Binary, _Unary, _is_scalar_shape
from ..ops.linalg import MatMulOp, _mm_shape
from ..ops.loss import SoftmaxCrossEntropyOp, SoftmaxCrossEntropyGradientOp
from ..ops.misc import OneHotOp, PlaceholderOp, _FillLike, SwapInOp, SwapOutOp
from ..ops.norm import BatchNormGradScaleOp, BatchNormOp
from ..ops.shape import AddBroadcastOp, ReduceSumOp, ReshapeOp, ReshapeGradientOp, SliceOp

FULL, ROW, SCALAR = 0, 1, 2
_BINARY = 32                       # instruction code of binary operator 0
_TAKES_NUMBER = (G.UN_ADDC, G.UN_MULC, G.UN_CDIV, G.UN_FILL)
MAX_IN, MAX_INS, MAX_SLOTS = 32, 64, 48
#: products of one launch, and what makes one small: the 128 x 64 tiles of one and of all, and K (longer sums are split)
MAX_GROUP, GROUP_TILES, GROUP_TILES_ALL, GROUP_K = 16, 16, 128, 480
#: rows of a column sum that is taken together with others
GROUP_ROWS = 512
#: value slots of a program over a tensor that does not fit in L2: more of them leave too few threads to cover DRAM
MAX_SLOTS_LARGE, LARGE = 12, 8 << 20


def _key(arr):
    """What two arrays share when element i of one belongs to element i of the other in memory order."""
    t = arr.t
    if t.is_contiguous():
        return ("rows", t.numel())
    return (arr.shape, arr.strides) if arr.is_dense() else None


def _row_stride(arr):
    """Of a matrix whose rows are contiguous, dense or a slice of wider ones; 0: another layout."""
    if arr.is_contiguous():
        return arr.shape[-1]
    return arr.strides[0] if len(arr.shape) == 2 and arr.strides[1] == 1 and arr.strides[0] >= arr.shape[1] else 0


def _code(node):
    op = node.op
    if isinstance(op, AddBroadcastOp):
        return _BINARY + G.BIN_ADD
    if isinstance(op, _FillLike):
        return G.UN_FILL
    if isinstance(op, _Binary):
        return _BINARY + op.gpu_code
    return op.gpu_code


def _constant(node):
    """The number an operator takes besides its operands, read in every step as the operator itself does."""
    if isinstance(node.op, _FillLike):
        return float(node.op.value)
    return 0.0 if node.const_attr is None else float(node.const_attr)


class Program(object):
    """Element-wise nodes collected so far (``members``, in order) and what they read from outside."""

    def __init__(self, key, numel):
        self.key, self.numel = key, numel
        self.members, self.values, self.inputs = [], {}, []      # values: node -> index of its instruction
        self.left, self.live = {}, 0         # member -> its readers outside; members that have such readers
        self.kinds, self.slot_of_input, self.cols = [], {}, 0

    def close(self, stored):
        """Assigns value slots (``stored``: the members whose results are read outside)."""
        last = {}
        for k, (node, ins) in enumerate(self.members):
            for ref in ins:
                last[ref] = k
        n_in = len(self.inputs)
        free, used = [], n_in
        where = {("in", j): j for j in range(n_in)}
        code, self.out = [], []
        self.constants = []                                 # (instruction, node) of those that take a number
        for k, (node, ins) in enumerate(self.members):
            op = _code(node)
            if op in _TAKES_NUMBER:
                self.constants.append((k, node))
            at = [where[ref] for ref in ins]
            for ref in dict.fromkeys(ins):
                if last[ref] == k:
                    free.append(where[ref])          # an instruction reads its operands before it writes
            if free:
                dst = free.pop()
            else:
                dst, used = used, used + 1
            where[("val", k)] = dst
            if ("val", k) not in last:
                free.append(dst)
            a = at[0] if at else 0
            code += [op, a, at[1] if len(at) > 1 else a, dst]
            self.out.append(node if node in stored else None)
        self.slots = max(used, 1)
        self.code = bytes(code)
        self.members = [m for m, _ in self.members]
        del self.values, self.slot_of_input, self.left      # needed while collecting only
        return self.slots

    def run(self, vals, arrays, stream):
        """False when an input is not laid out as planned (a feed may be): the caller runs the nodes one by one."""
        ptrs = []
        for node, kind in zip(self.inputs, self.kinds):
            v = vals[node]
            if kind == FULL:
                if _key(v) != self.key:
                    return False
            elif not v.is_contiguous():
                return False
            p = v.ptr
            if kind != SCALAR and p & 15:
                return False
            ptrs.append(p)
        outs = [arrays[n].ptr if n is not None else 0 for n in self.out]
        if any(p & 15 for p in outs):
            return False
        alpha = [0.0] * len(outs)
        for k, node in self.constants:
            alpha[k] = _constant(node)
        G.pointwise(ptrs, self.kinds, self.code, alpha, outs, self.slots, self.numel, self.cols, stream)
        return True


class StepPlan(object):
    def __init__(self, ex, fed):
        self.arrays = ex.node_to_arr_map
        self.shapes = ex.node_to_shape_map
        self.placeholders = [n for n in ex.topo_order if isinstance(n.op, PlaceholderOp) and n not in fed]
        self.evals = set(ex.eval_node_list)
        self.external = set(self.placeholders) | set(fed)
        self.kinds = {}                   # operator type -> _kind
        # place: how many nodes with effects stand before a node.  What a rule takes together must have the same number, or
        # one of its operands may be another by then.
        self.users, self.place, own, effects = {}, {}, {}, set()      # own: operator type -> nodes
        for n in ex.topo_order:
            self.place[n] = len(effects)
            if n not in self.external:
                own.setdefault(type(n.op), []).append(n)
                for i in n.inputs:
                    self.users.setdefault(i, []).append(n)
                if self._has_effects(n):
                    effects.add(n)

        def of(op):
            return [n for t, nodes in own.items() if issubclass(t, op) for n in nodes]
        losses = of(SoftmaxCrossEntropyOp)
        self.smooth, self.elided = {}, set()
        for n in losses:
            self._smooth_labels(n)
        self.sliced = {n for n in of(SliceOp) if self._is_sliced(n)}
        self.both = {}                           # gradient of a loss -> the loss that is computed with it
        for n in losses:
            self._loss_with_gradient(n)
        self.late = set(self.both.values())
        self.dense, self.stored = {}, set()      # product -> (its bias node or None, its ReLU or None), see _dense
        self.refused = {}                        # product -> what its launch does not take: 1 the ReLU, 2 the bias either
        for n in of(MatMulOp):
            self._dense(n)
        self.joined, self.inner = {}, set()      # addition -> the batch norm or the gradient that it is computed with; these
        for n in own.get(AddReluOp, ()):
            self._join(n)
        for n in own.get(AddOp, ()):
            self._add_gradients(n)
        self.root = {}                    # view -> the node whose array it looks at
        self.actions = []
        self.open = {}                    # key -> Program that still collects
        self.home = {}                    # node -> its open Program
        self.copies, self.copied = [], set()                     # (the same nodes twice)
        self.layouts = {n: (_key(a), a.t.numel()) for n, a in self.arrays.items()}
        self.group_of, self.queues, self.gone = {}, {}, set()    # ready operators that may share a launch, see _mates
        segment = []
        for n in ex.topo_order:
            if n in self.external:
                continue
            if n in effects:
                self._schedule(segment)
                segment = []
                self._flush_all()
                self.actions.append(("node", n))
            else:
                segment.append(n)
        self._schedule(segment)
        self._flush_all()
        del self.users, self.shapes, self.external, self.root, self.open, self.home, self.copies     # planning only
        del self.copied, self.layouts, self.group_of, self.queues, self.gone, self.kinds, self.stored, self.place

    def _kind(self, n):
        """What nodes of this operator type may become; "effects": they stay where they are."""
        op = type(n.op)
        kind = self.kinds.get(op)
        if kind is None:
            kind = "other"
            if not op.__module__.startswith("tsplit_b200.ops.") or issubclass(op, (SwapInOp, SwapOutOp)):
                kind = "effects"
            elif issubclass(op, (ReshapeOp, ReshapeGradientOp)):
                kind = "view"
            elif issubclass(op, BatchNormGradScaleOp):
                kind = "copy"
            elif issubclass(op, (_Binary, _Unary, _FillLike, AddBroadcastOp)):
                kind = "element"
            self.kinds[op] = kind
        return kind

    def _has_effects(self, n):
        return n.phase == "update" or self._kind(n) == "effects"

    # -- what a node is -------------------------------------------------------------------
    def _is_view(self, n):
        """Row-major reshapes of computed arrays (a result that the caller keeps stays an array of its own)."""
        if n in self.evals:
            return False
        src, arr = self.arrays.get(n.inputs[0]), self.arrays.get(n)
        return (src is not None and arr is not None and n.inputs[0] not in self.evals and src.t.is_contiguous()
                and arr.t.is_contiguous() and src.t.numel() == arr.t.numel())

    def _is_sliced(self, n):
        """Rows and columns of a value that is there from the start, for products, which take any row stride.  (The value
        may be a parameter: behind its update a view would show the new one.)"""
        users = self.users.get(n, ())
        return (n not in self.evals and n.inputs[0] in self.external and len(self.shapes[n]) == 2 and len(users) > 0
                and all(isinstance(u.op, MatMulOp) and not self._has_effects(u) and self.place[u] == self.place[n] for u in users))

    def _operands(self, n):
        """[(node, kind)] when ``n`` can be part of a program, else None."""
        if n not in self.layouts:
            return None
        key, numel = self.layouts[n]
        if key is None or numel == 0 or numel % 4:
            return None
        if isinstance(n.op, _FillLike):
            return []
        res, shapes, own = [], self.shapes, self.shapes[n]
        for j, i in enumerate(n.inputs):
            shape, at = shapes[i], self.layouts.get(i)
            if shape == own and (at is None or at[0] == key):
                res.append((i, FULL))
            elif isinstance(n.op, AddBroadcastOp) and j == 1:
                cols = own[-1]
                if key[0] != "rows" or cols % 4 or shape[-1] != cols or ndarray._numel(shape) != cols:
                    return None
                res.append((i, ROW))
            elif _is_scalar_shape(shape) and isinstance(n.op, _Binary):
                res.append((i, SCALAR))
            else:
                return None
        return res

    def _smooth_labels(self, ce):
        """When ``ce``'s labels are ``one_hot(ids) * a + b`` (any number of constants, reshapes that keep the classes)
        and nothing but cross-entropies over them reads any of it: remember ids and the operators on the way."""
        labels = cur = ce.inputs[1]
        chain, consts = [], []
        while True:
            if cur in self.external or cur in self.evals or self._has_effects(cur) or self.arrays.get(cur) is None:
                return
            chain.append(cur)
            if isinstance(cur.op, OneHotOp):
                break
            if isinstance(cur.op, (AddConstOp, MulConstOp)):
                consts.append(cur)
            elif not (isinstance(cur.op, ReshapeOp) and self.arrays[cur].t.is_contiguous()):
                return
            cur = cur.inputs[0]
            if tuple(self.shapes[cur])[-1:] != tuple(self.shapes[labels])[-1:]:
                return
        readers = self.users.get(labels, [])
        if len(self.shapes[labels]) != 2 or not all(
                isinstance(u.op, (SoftmaxCrossEntropyOp, SoftmaxCrossEntropyGradientOp)) and u.inputs[1] is labels
                and u.inputs.count(labels) == 1 for u in readers):
            return
        if any(u not in chain for m in chain[1:] for u in self.users.get(m, ())):
            return
        if len({self.place[u] for u in chain + readers}) > 1:       # an update may change the ids in between
            return
        self.elided.update(chain)
        for u in readers:
            self.smooth[u] = (cur.inputs[0], consts[::-1], chain[::-1])

    def _loss_with_gradient(self, loss):
        """When nobody needs ``loss`` before its one gradient is due (a seed of ones takes its shape only), and no update of
        its logits or labels stands between the two."""
        logits, labels = loss.inputs
        grads = [u for u in self.users.get(logits, ()) if isinstance(u.op, SoftmaxCrossEntropyGradientOp)
                 and u.inputs[0] is logits and u.inputs[1] is labels]
        others = [u for u in self.users.get(logits, ()) if isinstance(u.op, SoftmaxCrossEntropyOp) and u.inputs[1] is labels]
        if (len(grads) == 1 and len(others) == 1 and self.place[grads[0]] == self.place[loss]
                and all(isinstance(u.op, _FillLike) for u in self.users.get(loss, ()))
                and (loss in self.smooth) == (grads[0] in self.smooth) and not self._has_effects(loss)
                and not self._has_effects(grads[0]) and self.arrays.get(loss) is not None
                and self.arrays.get(grads[0]) is not None):
            self.both[grads[0]] = loss

    def _dense(self, product):
        """``product + row`` that nothing else reads the product of, and the one ReLU of the result (or of the product
        itself): the product's launch can store them.  The row is there from the start, a parameter: an addition behind its
        update has to read the new one."""
        result, bias, readers = product, None, self.users.get(product, [])
        if (len(readers) == 1 and isinstance(readers[0].op, AddBroadcastOp) and readers[0].inputs[0] is product
                and product not in self.evals and not self._has_effects(readers[0]) and self.place[readers[0]] == self.place[product]):
            row = readers[0].inputs[1]
            cols = self.shapes[product][-1]
            if row in self.external and row is not product and tuple(self.shapes[row]) == (cols,):
                result = bias = readers[0]
        relus = [u for u in self.users.get(result, ())
                 if isinstance(u.op, ReluOp) and not self._has_effects(u) and self.place[u] == self.place[product]]
        relu = relus[0] if len(relus) == 1 else None
        made = [n for n in (bias, relu) if n is not None]
        own = self.arrays.get(product)
        if made and own is not None and own.is_contiguous() and all(
                self.arrays.get(n) is not None and self.arrays[n].is_contiguous()
                and tuple(self.shapes[n]) == tuple(self.shapes[product]) for n in made):
            self.dense[product] = (bias, relu)
            self.stored.update(made)

    def _join(self, n):
        """``relu(a + batch_norm(x))`` that alone reads the batch norm (its gradient does not): one apply pass for both."""
        for b in sorted(set(n.inputs), key=lambda i: -i.id):
            if (type(b.op) is BatchNormOp and b not in self.external and b not in self.evals and self.users.get(b) == [n]
                    and n.inputs.count(b) == 1 and self.place[b] == self.place[n] and not self._has_effects(n)
                    and self.arrays.get(b) is not None and self.arrays.get(n) is not None
                    and all(tuple(self.shapes[i]) == tuple(self.shapes[n]) for i in n.inputs)):
                self.joined[n] = b
                self.inner.add(b)
                return

    def _add_gradients(self, n):
        """The sum of two convolutions' gradients that alone reads them, one of stride 2: the other one's result is written
        where the sum goes, and this one adds to it."""
        def alone(i):
            return (type(i.op) is Conv2dGradDataOp and i not in self.external and i not in self.evals and self.users.get(i) == [n]
                    and self.place[i] == self.place[n] and i not in self.inner
                    and self.arrays.get(i) is not None and tuple(self.shapes[i]) == tuple(self.shapes[n]))
        a, b = n.inputs
        if a is b or self.arrays.get(n) is None or self._has_effects(n) or not (alone(a) and alone(b)):
            return
        late = b if b.attrs["stride"] == 2 else a
        first = a if late is b else b
        if late.attrs["stride"] == 2 and self.arrays[first].same_layout(self.arrays[n]):
            self.joined[n] = late
            self.inner.add(late)
            self.arrays[first] = self.arrays[n]

    # -- scheduling ------------------------------------------------------------------------
    def _schedule(self, nodes):
        inside = set(nodes)
        waits = {n: sum(1 for i in set(n.inputs) if i in inside) for n in nodes}
        users = self.users
        # ready nodes: those that cost no launch of their own, the others, and of these the column sums that may wait
        light, heavy, sums, waiting = [], [], [], 0
        self.queues, self.gone = {}, set()

        def ready(n):
            nonlocal waiting
            cls, ops = "elided" if n in self.elided or n in self.stored else self._kind(n), None
            if n in self.inner:
                cls = "elided"
            elif n in self.joined:
                cls = None
            elif cls == "element":
                ops = self._operands(n)
                cls = None if ops is None else cls
            elif n in self.sliced:
                cls = "slice"
            elif cls == "other" or cls == "view" and not self._is_view(n):
                cls = None
            if cls:
                heapq.heappush(light, (n.id, n, cls, ops))
                return
            group = self.group_of[n] = self._group(n)
            may_wait = group is not None and group[0] == ("sums",)
            heapq.heappush(sums if may_wait else heavy, (n.id, n))
            waiting += may_wait
            if group:
                heapq.heappush(self.queues.setdefault(group[0], []), (n.id, n, group[1]))

        def done(n):
            for u in set(users.get(n, ())):
                if u in waits:
                    waits[u] -= 1
                    if waits[u] == 0:
                        ready(u)
        for n in nodes:
            if waits[n] == 0:
                ready(n)
        while light or heavy or sums:
            if light:
                _, n, cls, ops = heapq.heappop(light)
                if cls == "elided":
                    pass
                elif cls == "slice":
                    self.actions.append(("slice", n))
                elif cls == "view":
                    self._view(n)
                elif cls == "copy":
                    self._need(n.inputs[0])
                    self.copies.append(n)
                    self.copied.add(n)
                else:
                    self._collect(n, ops)
            else:
                _, n = heapq.heappop(heavy if heavy and waiting < MAX_GROUP else sums or heavy)
                if n in self.gone:
                    continue
                taken = self._mates(n)
                if self.group_of[n] and self.group_of[n][0] == ("sums",):
                    waiting -= len(taken)
                for m in taken:
                    for i in m.inputs:
                        self._need(i)
                if n in self.joined:
                    for i in self.joined[n].inputs:
                        self._need(i)
                if n in self.smooth:
                    self._need(self.smooth[n][0])
                self.actions.append((self.group_of[n][0][0], taken) if len(taken) > 1 else
                                    ("smooth", n) if n in self.smooth else
                                    ("loss", n) if n in self.both or n in self.late else
                                    ("join", n) if n in self.joined else
                                    ("products", taken) if n in self.dense or not self.sliced.isdisjoint(n.inputs) else
                                    ("node", n))
                for m in taken[1:]:
                    done(m)
            done(n)

    def _group(self, n):
        """(kind, blocks) of an operator small enough to share a launch with others of its kind, else None."""
        if self.arrays.get(n) is None:
            return None
        if isinstance(n.op, MatMulOp):
            ta, tb = n.attrs["trans_A"], n.attrs["trans_B"]
            m, c, k = _mm_shape(self.shapes[n.inputs[0]], self.shapes[n.inputs[1]], ta, tb)
            tiles = -(-m // 128) * -(-c // 64)
            return (("products", bool(ta), bool(tb)), tiles) if tiles <= GROUP_TILES and k <= GROUP_K else None
        if isinstance(n.op, ReduceSumOp):
            shape, axes = self.shapes[n.inputs[0]], n.attrs["axes"]
            if len(shape) == 2 and list(axes) == [0] and 1 < shape[0] <= GROUP_ROWS and shape[1] <= 1024:
                return ("sums",), 1
        return None

    def _mates(self, n):
        """``n`` and the operators that are ready with it and go into the same launch: the next ones of its kind, as long
        as they fit.  They stay in the heap of ready operators and are passed over there (``gone``)."""
        taken, own = [n], self.group_of[n]
        self.gone.add(n)
        if own:
            kind, blocks = own
            queue = self.queues[kind]
            while queue and len(taken) < MAX_GROUP:
                _, m, more = queue[0]
                if m not in self.gone:
                    if blocks + more > GROUP_TILES_ALL:
                        break
                    taken.append(m)
                    self.gone.add(m)
                    blocks += more
                heapq.heappop(queue)
        return taken

    def _view(self, n):
        src = n.inputs[0]
        self.root[n] = self.root.get(src, src)
        base, own = self.arrays[src], self.arrays[n]
        # (with the strides of the array it replaces: kernels read those of dimensions of one element, too)
        view = ndarray.NDArray(base.t.as_strided(own.shape, own.strides, base.t.storage_offset()), base.ctx, owns=False)
        view._base = base                  # the bytes live as long as anything looks at them
        self.arrays[n] = view
        self.actions.append(("view", n))

    def _need(self, i):
        """``i``'s array is read by something outside its program: run that now."""
        i = self.root.get(i, i)
        if i in self.home:
            self._flush(self.home[i])
        elif i in self.copied:
            self._flush_copies()

    def _collect(self, n, operands):
        key, numel = self.layouts[n]
        home, prog, cols = self.home, self.open.get(key), 0
        operands = [(self.root.get(i, i), kind) for i, kind in operands]
        for r, kind in operands:
            if kind != FULL or prog is None or home.get(r) is not prog:
                self._need(r)              # computed by another program, or read in another way than its values lie
            if kind == ROW:
                cols = self.shapes[n][-1]
        prog = self.open.get(key)          # (the call above may have run it)
        if prog is not None:
            new = len({r for r, _ in operands if home.get(r) is not prog})
            limit = MAX_SLOTS_LARGE if numel >= LARGE else MAX_SLOTS
            if (len(prog.inputs) + new > min(MAX_IN, limit - 4) or len(prog.members) >= MAX_INS
                    or (cols and prog.cols and prog.cols != cols) or self._too_many_slots(prog, n, limit)):
                self._flush(prog)
                prog = None
        if prog is None:
            prog = self.open[key] = Program(key, numel)
        refs = []
        for r, kind in operands:
            if home.get(r) is prog:
                refs.append(("val", prog.values[r]))
                continue
            slot = prog.slot_of_input.get((r, kind))
            if slot is None:
                slot = prog.slot_of_input[(r, kind)] = len(prog.inputs)
                prog.inputs.append(r)
                prog.kinds.append(kind)
            refs.append(("in", slot))
        prog.cols = prog.cols or cols
        prog.values[n] = len(prog.members)
        prog.members.append((n, refs))
        home[n] = prog
        for i in n.inputs:
            if i in prog.left:
                prog.left[i] -= 1
                prog.live -= not prog.left[i]
        readers = prog.left[n] = len(self.users.get(n, ()))
        prog.live += readers > 0

    @staticmethod
    def _too_many_slots(prog, n, limit):
        """After one more member: every value still read later holds one."""
        most = len(prog.inputs) + prog.live + 3
        return most > limit and most - sum(          # (less those that are read by nobody after n)
            1 for i in set(n.inputs) if prog.left.get(i) == n.inputs.count(i)) > limit

    def _flush(self, prog):
        del self.open[prog.key]
        members = [m for m, _ in prog.members]
        for m in members:
            del self.home[m]
        # (views count as readers outside: theirs are)
        stored = {m for m in members if m in self.evals or prog.left[m]}
        if len(members) == 1 or prog.close(stored) > MAX_SLOTS:
            self.actions += [("node", m) for m in members]
        else:
            self.actions.append(("program", prog))

    def _flush_copies(self):
        for lo in range(0, len(self.copies), 64):
            self.actions.append(("copies", self.copies[lo:lo + 64]))
        self.copies, self.copied = [], set()

    def _flush_all(self):
        for prog in list(self.open.values()):
            self._flush(prog)
        self._flush_copies()

    # -- execution --------------------------------------------------------------------------
    def run(self, ex, vals):
        for n in self.placeholders:
            vals[n] = ex._placeholder_value(n)
        for n in self.elided:              # (for those who walk all values, as a per-operator timing does)
            vals[n] = self.arrays[n]
        stream = ex.stream
        made = set()                       # labels that had to be made after all: once a step, however many read them
        for what, x in self.actions:
            if what == "node":
                self._node(x, vals, stream)
            elif what == "view":
                vals[x] = self.arrays[x]
            elif what == "slice":
                vals[x] = self._slice(x, vals[x.inputs[0]], vals, stream)
            elif what in ("loss", "smooth"):
                if x in self.late:
                    vals[x] = self.arrays[x]         # (a seed of ones takes its shape)
                elif x in self.both:
                    self._loss(x, vals, stream, made)
                else:
                    self._smooth(x, vals, stream, made)
            elif what == "products":
                self._products(x, vals, stream)
            elif what == "sums":
                self._sums(x, vals, stream)
            elif what == "join":
                self._joined(x, vals, stream)
            elif what == "program":
                if x.run(vals, self.arrays, stream):
                    for m in x.members:
                        vals[m] = self.arrays[m]
                else:
                    for m in x.members:
                        self._node(m, vals, stream)
            else:
                src = [n.inputs[0].state[n.op.key] for n in x]
                dst = [self.arrays[n] for n in x]
                if all(a.is_dense() and a.same_layout(b) for a, b in zip(src, dst)):
                    G.multi_copy(src, dst, stream)
                    for n in x:
                        vals[n] = self.arrays[n]
                else:
                    for n in x:
                        self._node(n, vals, stream)

    def _slice(self, n, src, vals, stream):
        """A view of ``src`` that products read in place, or else ``n``'s own array with the values in it."""
        begin, own = n.attrs["begin"], self.arrays[n]
        if src.is_contiguous() and src.shape[1] % 4 == 0 and own.is_contiguous():
            at = src.t.storage_offset() + begin[0] * src.shape[1] + begin[1]
            view = ndarray.NDArray(src.t.as_strided(own.shape, (src.shape[1], 1), at), src.ctx, owns=False)
            view._base = src
            if view.ptr % 16 == 0:
                return view
        n.op.compute(n, [src], own, False, stream)
        return own

    def _products(self, nodes, vals, stream):
        ta, tb = nodes[0].attrs["trans_A"], nodes[0].attrs["trans_B"]
        if (self.refused.get(nodes[0], 0) < 2 and any(n in self.dense for n in nodes)
                and self._dense_products(nodes, ta, tb, vals, stream)):
            return
        items, alone = [], []
        for n in nodes:
            a, b, out = vals[n.inputs[0]], vals[n.inputs[1]], self.arrays[n]
            if _row_stride(a) and _row_stride(b) and out.is_contiguous() and G.gemm_group_takes(a, b):
                items.append((n, (a, b, out) + _mm_shape(a.shape, b.shape, ta, tb)))
            else:
                alone.append(n)            # (a row of 10 classes needs padding, which a group does not do)
        one = len(items) == 1 and not self.sliced.isdisjoint(items[0][0].inputs)
        if (len(items) > 1 and G.gemm_group([i for _, i in items], ta, tb, stream)
                or one and G.gemm_dense([i + (None, None) for _, i in items], ta, tb, stream)):
            for n, _ in items:
                vals[n] = self.arrays[n]
        else:
            alone = nodes
        for n in alone:
            self._node(n, vals, stream)
        for n in nodes:
            for m in self.dense.get(n, ()):
                if m is not None:
                    self._node(m, vals, stream)

    def _dense_products(self, nodes, ta, tb, vals, stream):
        """The products with what their launches store besides; False: not taken.  (The array of a product whose bias is
        added there is not written; the sums alone would be read by nobody.)"""
        items = []
        for n in nodes:
            bias, relu = self.dense.get(n, (None, None))
            a, b = vals[n.inputs[0]], vals[n.inputs[1]]
            row = vals[bias.inputs[1]] if bias is not None else None
            if not (_row_stride(a) and _row_stride(b) and (row is None or row.is_contiguous())):
                return False
            items.append((a, b, self.arrays[n if bias is None else bias]) + _mm_shape(a.shape, b.shape, ta, tb)
                         + (row, None if relu is None else self.arrays[relu]))
        if len(items) > 1 and not all(G.gemm_group_takes(*i[:2]) for i in items):
            return False
        first, late = nodes[0], []
        has_relu, has_bias = (any(i[j] is not None for i in items) for j in (7, 6))
        taken = first not in self.refused and G.gemm_dense(items, ta, tb, stream)
        if not taken and has_relu and has_bias and self.refused.get(first, 1) < 2:
            # a ReLU is stored by small products only: without it
            self.refused[first] = 1
            late = [self.dense[n][1] for n in nodes if n in self.dense and self.dense[n][1] is not None]
            taken = G.gemm_dense([i[:7] + (None,) for i in items], ta, tb, stream)
        if not taken:
            self.refused[first] = 2
            return False
        for n in nodes:
            for m in (n,) + self.dense.get(n, ()):
                if m is not None:
                    vals[m] = self.arrays[m]
        for m in late:
            self._node(m, vals, stream)
        return True

    def _sums(self, nodes, vals, stream):
        items = [(vals[n.inputs[0]], self.arrays[n]) for n in nodes]
        if all(x.is_contiguous() and y.is_contiguous() for x, y in items) and G.colsum_group(items, stream):
            for n in nodes:
                vals[n] = self.arrays[n]
        else:
            for n in nodes:
                self._node(n, vals, stream)

    def _joined(self, n, vals, stream):
        """(The inner node's own array is not written: nobody else reads it.)"""
        inner, out = self.joined[n], self.arrays[n]
        other = vals[n.inputs[0] if n.inputs[1] is inner else n.inputs[1]]
        ins = [vals[i] for i in inner.inputs]
        if (inner.op.forward_add(inner, ins, other, out, stream) if type(n.op) is AddReluOp else inner.op.add_to(inner, ins, out, stream)):
            vals[inner], vals[n] = self.arrays[inner], out
        else:
            self._node(inner, vals, stream)
            self._node(n, vals, stream)

    def _loss(self, n, vals, stream, made):
        """A gradient and the loss that waited for it."""
        loss = self.both[n]
        x, g, out, grad = vals[n.inputs[0]], vals[n.inputs[2]], self.arrays[loss], self.arrays[n]
        if x.is_contiguous() and grad.is_contiguous():
            if n in self.smooth:
                ids = vals[self.smooth[n][0]]
                ok = ids.is_contiguous() and G.softmax_ce_both_smooth(x, ids, *self._on_off(n), g, out, grad, stream)
            else:
                labels = vals[n.inputs[1]]
                ok = labels.is_contiguous() and G.softmax_ce_both(x, labels, g, out, grad, stream)
            if ok:
                vals[loss], vals[n] = out, grad
                return
        for m in (loss, n):
            if m in self.smooth:
                self._smooth(m, vals, stream, made)
            else:
                self._node(m, vals, stream)

    def _on_off(self, n):
        """What the operators of smoothed labels make of a one and of a zero."""
        on, off = np.float32(1), np.float32(0)
        for m in self.smooth[n][1]:
            c = np.float32(_constant(m))
            on, off = (on * c, off * c) if isinstance(m.op, MulConstOp) else (on + c, off + c)
        return float(on), float(off)

    def _smooth(self, n, vals, stream, made):
        ids, _, chain = self.smooth[n]
        on, off = self._on_off(n)
        x, i, out = vals[n.inputs[0]], vals[ids], self.arrays[n]
        ok = x.is_contiguous() and i.is_contiguous() and out.is_contiguous()
        if ok and isinstance(n.op, SoftmaxCrossEntropyOp):
            ok = G.softmax_ce_smooth(x, i, on, off, out, stream)
        elif ok:
            ok = G.softmax_ce_grad_smooth(x, i, on, off, vals[n.inputs[2]], out, stream)
        if ok:
            vals[n] = out
            return
        for m in chain:
            if m not in made:
                self._node(m, vals, stream)
        made.update(chain)
        self._node(n, vals, stream)

    def _node(self, n, vals, stream):
        for i in n.inputs:
            if i in self.sliced and not vals[i].is_contiguous():       # an operator that reads whole arrays only
                i.op.compute(i, [vals[i.inputs[0]]], self.arrays[i], False, stream)
                vals[i] = self.arrays[i]
        out = self.arrays.get(n)
        n.op.compute(n, [vals[i] for i in n.inputs], out, False, stream)
        vals[n] = out
