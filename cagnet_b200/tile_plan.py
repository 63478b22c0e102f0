"""Choosing the dense tiles of a normalised CSR block and cutting them out (index work, once per block).

With rows and columns ranked by degree, a power-law block concentrates its nonzeros in a corner whose density falls
off smoothly; the tiles of 256 rows x 64 columns that are full enough go to the tensor cores as bit matrices
(csrc/tile_core.cu), everything else stays sparse.  Unlike one rectangle (core_select.choose_core) the tiles follow the
shape of that corner: hub rows keep far more columns than ordinary ones.  The reference has no counterpart: its SpMM hands
the whole block to cuSPARSE (sparse-extension/sparse_coo_tensor.cu:198-226).
"""
import torch

ROWS, COLS, WORDS = 256, 64, 512          # a tile and the 32-bit words of its bit matrix
BLOCKS = 148                              # persistent thread blocks of the multiply, one per SM

# What a tile has to beat, in nonzeros.  A row panel costs its multiply the pass over 256 rows of C (as much as PANEL_COST
# tiles' products) and a 64-column block the three-term operand that is written and read once per multiply: tiles of panels
# or column blocks whose nonzeros beyond the bar do not add up to these are left sparse.  (Measured per tile: 0.33 us of one
# SM at width 16, 7.3 us at width 602; per gathered nonzero 1 ns and 25 ns; per panel 1 us and 5 us.)
PANEL_NNZ, KB_NNZ = 1000, 600
PANEL_COST = 3.0


def ranks(deg):
    """Order by degree, highest first (ties by index), and each index's place in it (int32)."""
    order = torch.argsort(deg, descending=True, stable=True)
    place = torch.empty(deg.numel(), dtype=torch.int32, device=deg.device)
    place[order] = torch.arange(deg.numel(), dtype=torch.int32, device=deg.device)
    return order, place


def select(counts, bar):
    """bool mask over the (row panel, column block) counts: tiles of at least `bar` nonzeros in panels and column blocks
    that are worth their fixed cost."""
    on = counts >= bar
    extra = (counts - bar).clamp_min(0)
    for _ in range(2):
        on &= ((extra * on).sum(1) >= PANEL_NNZ)[:, None]
        on &= ((extra * on).sum(0) >= KB_NNZ)[None, :]
    return on


def shares(panel_of, panel_ptr, blocks=BLOCKS):
    """(first tile of every block's share, list of cut panels): consecutive shares of about equal cost, none empty."""
    tiles = panel_of.numel()
    blocks = min(blocks, tiles)
    cost = torch.arange(1, tiles + 1, dtype=torch.float64, device=panel_of.device) + PANEL_COST * (panel_of + 1).double()
    at = torch.arange(blocks + 1, dtype=torch.float64, device=panel_of.device) * (float(cost[-1]) / blocks)
    step = torch.arange(blocks + 1, device=panel_of.device)
    first = torch.searchsorted(cost, at)
    first[0], first[-1] = 0, tiles
    first = torch.cummax(first - step, 0)[0] + step                   # at least one tile each
    first = torch.minimum(first, tiles - blocks + step)
    starts, ends = first.tolist(), panel_ptr.tolist()
    held = torch.searchsorted(panel_ptr, first, right=True).sub(1).tolist()
    cuts = {}
    for i in range(1, blocks):
        p = held[i]
        if ends[p] < starts[i]:                                        # the boundary lies inside panel p
            cuts[p] = (cuts.get(p, (i - 1,))[0], i + 1)
    return first.int(), [(p, a, b, 0) for p, (a, b) in cuts.items()]


class TilePlan:
    """Device arrays of the chosen tiles as `cagnet_block` names them."""

    def __init__(self, on, order_r, order_c, lim_r, lim_c, row_scale):
        dev = on.device
        panels, kbs = on.size(0), on.size(1)
        active = torch.nonzero(on.flatten()).flatten()
        panel, kb = torch.div(active, kbs, rounding_mode="floor"), active % kbs
        used_p, used_k = torch.unique(panel), torch.unique(kb)
        self.tiles = int(active.numel())
        self.panels, self.tile_kbs = int(used_p.numel()), int(used_k.numel())
        self.tile_of = torch.full((panels * kbs,), -1, dtype=torch.int32, device=dev)
        self.tile_of[active] = torch.arange(self.tiles, dtype=torch.int32, device=dev)
        new_p = torch.zeros(panels, dtype=torch.int64, device=dev)
        new_p[used_p] = torch.arange(self.panels, device=dev)
        new_k = torch.zeros(kbs, dtype=torch.int64, device=dev)
        new_k[used_k] = torch.arange(self.tile_kbs, device=dev)
        self.tile_kb = new_k[kb].int()
        ptr = torch.zeros(self.panels + 1, dtype=torch.int64, device=dev)
        ptr[1:] = torch.cumsum(torch.bincount(new_p[panel], minlength=self.panels), 0)
        self.panel_ptr = ptr.int()
        self.cta_ptr, cuts = shares(new_p[panel], ptr)
        self.ctas, self.joins = int(self.cta_ptr.numel()) - 1, len(cuts)
        self.join_list = torch.tensor(cuts or [(0, 0, 0, 0)], dtype=torch.int32, device=dev)

        def pick(order, limit, size, used):
            full = torch.full((size,), -1, dtype=torch.int32, device=dev)
            full[:limit] = order[:limit].int()
            return full.view(used[0], used[1])[used[2]].flatten().contiguous()

        self.tile_cols = pick(order_c, lim_c, kbs * COLS, (kbs, COLS, used_k))
        self.panel_rows = pick(order_r, lim_r, panels * ROWS, (panels, ROWS, used_p))
        self.panel_scale = torch.where(self.panel_rows >= 0, row_scale[self.panel_rows.clamp_min(0).long()],
                                       torch.zeros((), device=dev)).contiguous()
        self.tile_bits = torch.zeros(self.tiles * WORDS, dtype=torch.int32, device=dev)
