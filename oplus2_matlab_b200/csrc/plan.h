// plan.h -- device execution plans (not installed).
#pragma once

#include <memory>
#include <vector>

#include "internal.h"

namespace op2b {

// The reference's execution plan (common/op_lib_core.h:122-150), built on the
// device by build_plan() and kept there.  Arrays follow the reference's
// definitions exactly; `pub` is the op_plan view handed to callers of
// op_plan_get (device pointers except ncolblk and nindirect).
struct DevPlan {
  // cache key (common/op_lib_core.c:632-659)
  std::string name;
  op_set set = nullptr;
  int part_size = 0, nargs = 0, ninds = 0;
  std::vector<op_dat> dats;
  std::vector<op_map> maps;
  std::vector<int> idxs, inds;
  std::vector<op_access> accs;

  int bsize = 0, nblocks = 0, ncolors = 0, nshared = 0;
  int *d_nthrcol = nullptr, *d_thrcol = nullptr, *d_offset = nullptr, *d_nelems = nullptr;
  int *d_ind_offs = nullptr, *d_ind_sizes = nullptr, *d_blkmap = nullptr;
  int *d_blkcol = nullptr;  // colour of each block
  std::vector<int *> d_ind_maps;
  std::vector<short *> d_loc_maps;
  std::vector<int> nindirect, ncolblk, colstart;  // host
  std::vector<int> nthrcol_h;                     // host copy (for diagnostics)
  double transfer = 0, transfer2 = 0, transfer3 = 0;
  float avg_thread_colours = 0;
  int max_thread_colours = 0;
  op_plan pub;
  std::vector<int *> pub_ind_maps;
  std::vector<short *> pub_loc_maps;
  int count = 0;
};

// Owner-computes ("gather") plan for one group of OP_INC arguments that
// increment the same dataset: for every target element, the list of
// (element, slot) contributions in ascending order, slot = position of the
// argument inside the group.  This is the order of the sequential back-end
// (common/op_seq.h:26-57, element loop outermost, arguments in kernel order).
struct GatherPlan {
  op_set set = nullptr;           // loop set
  op_dat dat = nullptr;           // incremented dataset
  std::vector<op_map> maps;       // per slot
  std::vector<int> idxs;          // per slot
  int nslots = 0;
  int ntarget = 0;                // size of dat->set
  int nactive = 0;                // targets with at least one contribution
  int *d_row = nullptr;           // [nactive + 1] offsets into d_keys
  int *d_keys = nullptr;          // [set->size * nslots] element * nslots + slot
  int *d_active = nullptr;        // [nactive] target ids, nullptr when all active
  int max_row = 0;
  // CTA tiles for the contribution-parallel kernels: tile b owns the
  // targets whose first contribution lies in [kTile*b, kTile*(b+1)), i.e.
  // targets [d_tile_first[b], d_tile_first[b+1]); [ntiles + 1] entries
  int ntiles = 0;
  int *d_tile_first = nullptr;
  long long nkeys = 0;
  // per-element contribution buffer of the two-pass kernels, allocated on
  // first use (outside any graph capture) and kept with the plan
  void *d_contrib = nullptr;
  size_t contrib_bytes = 0;
  bool unsuited = false;  // none of the arrays are there: Make::kTry gave up
};

// How far the finders of plans that a loop can do without may go: kFind returns
// what is there (in a capture, which cannot make them); kTry makes it, but
// reports no error and gives up, once and for all, on targets of more than
// kMaxSlotWidth contributions and where there is no room; kBuild makes it or
// reports an error.
enum class Make { kFind, kTry, kBuild };

// contributions per CTA tile of the contribution-parallel gather kernels
constexpr int kTile = 256;

// Fixed-width (ELL) contribution lists for an edge loop `a` with two
// increment arguments (slot 0 adds the edge's value, slot 1 subtracts it),
// optionally followed by a loop `b` with one (adds): the kernels store one
// value per edge of a in v[0, na), one per element of b in v[na, na+nb),
// and -0.0 in v[na+nb].  Target t owns entries ell[t*width, (t+1)*width):
// (index << 1 | negate) of its contributions, a's in a's ascending order
// then b's in b's order, padded with (na+nb) << 1.  Adding the entries in
// list order is the order of the sequential back-end running a then b;
// -0.0 is the exact identity of IEEE addition and r + (-v) equals r - v.
struct ChainSched;  // airfoil.cu: the persistent chain's work queue over these lists
struct TilePlan;    // airfoil.cu: the tiled chain's per-tile flux lists
struct SlotPlan {
  const GatherPlan *a = nullptr, *b = nullptr;
  int ntarget = 0;
  int width = 0;            // max contributions of one target
  int na = 0, nb = 0;       // elements of a and b
  int *d_ell = nullptr;     // [ntarget * width]
  void *d_buf = nullptr;    // the (na + nb + 1) values, allocated by the loop
  size_t buf_bytes = 0;
  bool no_room = false;  // Make::kTry found no room for the lists or the values
  ChainSched *chain = nullptr;  // built by the first persistent chain launch
  bool chain_unsuited = false;  // a cell tile reads too many flux tiles for it
  // the edges of a in the order the flux pass takes them (get_flux_order)
  struct Order {
    op_map mx = nullptr, mq = nullptr;  // the maps of the edges' nodes and cells
    op_dat x = nullptr;                 // the nodes' coordinates
    int4 *d_rows = nullptr;  // [na] the edges' rows of them: two nodes, two cells
    int *d_ell = nullptr;    // the lists, with the places of the edges' values
    // distinct cells of a sample of the order, and of the loop's own: rows and
    // lists hold the loop's order where that is no better (k_order_lists)
    unsigned long long *d_cells = nullptr;
    long long passes = 0;    // flux passes in the loop's order
    bool tried = false;
  };
  std::vector<std::unique_ptr<Order>> orders;
  bool scattered = false;  // a's elements, in order, reach targets without locality
  struct Coloured {  // get_coloured_lists
    const DevPlan *p, *pb;
    const Order *o;
    int nt, nbt, *d_ell;
  };
  std::vector<Coloured> coloured;
  TilePlan *tile = nullptr;     // built by the first tiled chain launch
  bool tile_unsuited = false;   // no tile size fits shared memory
};
// free a slot plan's persistent-chain queue and tile plan (airfoil.cu)
void release_chain_sched(SlotPlan *sp);
void release_tile_plan(SlotPlan *sp);

// A slot plan's lists in the order of the two-level colouring of a (plan p, nt
// threads per block) and b (pb, nbt; nullable): by block colour, then by
// strip of nt elements of the block, thread colour and slot, b's after a's;
// entry index << 2 | last of its block << 1 | negate, -1 past the end.
// o: when the flux pass has an order of its own.
// Device memory kept with the slot plan; nullptr when the indices do not fit,
// when there is no room, or when they are not there and a capture is under way,
// which cannot make them.
const int *get_coloured_lists(SlotPlan *sp, const SlotPlan::Order *o, const DevPlan *p, int nt,
                              const DevPlan *pb, int nbt);

// Find or build the flux pass's order of a's edges, whose nodes and cells are
// columns 0 and 1 of the dim-2 maps mx and mq and whose nodes have the dataset
// x (two reals: taken for coordinates when the numbering has no locality);
// nullptr: the loop's own order, or a capture that comes before it is built.
// after: the order may be made now, if this is at least that many passes after
// the first; < 0: only one that is there.  Values of a flux pass that has run are
// listed in the order that it took, so only a caller about to run one may make it
const SlotPlan::Order *get_flux_order(SlotPlan *sp, op_map mx, op_map mq, op_dat x,
                                      long long after);
// at the start of a capture, which is replayed often and cannot make them, and
// of the autotuner's timings
void make_flux_orders();
// the orders made, and those that the sample kept (waits; -1 in a capture)
int flux_orders(int *kept);

// widest list the fold kernels accept
constexpr int kMaxSlotWidth = 8;

// Find or build the lists of a (two slots) and b (nullable, one slot);
// nullptr when some target has more than kMaxSlotWidth contributions or the
// padding would more than double the lists (the caller then uses the CSR
// fold).
SlotPlan *get_slot_plan(const GatherPlan *a, const GatherPlan *b, Make make = Make::kBuild);

// Find or build the reference-compatible plan (device resident).
DevPlan *get_plan(char const *name, op_set set, int part_size, int nargs, const op_arg *args,
                  int ninds, const int *inds);
// the call that found it did not use it: op_plan's count of uses as before
void plan_unused(DevPlan *p);
// Find or build the gather plan for the INC args listed in slots (all on
// the same dat).
GatherPlan *get_gather_plan(op_set set, const op_arg *args, const std::vector<int> &slots,
                            Make make = Make::kBuild);
// Device validation of a plan; returns the number of violations.
long validate_plan(const DevPlan &p);

// device-wide exclusive scan of n ints (in place allowed); returns the total
long long exclusive_scan(const int *d_in, int *d_out, int n, cudaStream_t s);
// the same, queued only (no total, no host wait)
void exclusive_scan_nosync(const int *d_in, int *d_out, int n, cudaStream_t s);

}  // namespace op2b
