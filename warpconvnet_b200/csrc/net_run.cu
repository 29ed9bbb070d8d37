// A network's convolutions enqueued by one call.  From Python each launch costs 8-10 us of host time (argument
// objects, an output allocation), which for scenes of up to 150 000 voxels is more than the kernel takes; here it is the
// launch alone.
#include "wcn_common.cuh"

namespace {

template <typename P> P at(const wcn_net_buffer* buffers, int b, int col) {
  return b < 0 ? nullptr : reinterpret_cast<P>((char*)buffers[b].data + (int64_t)col * 2);
}

bool valid(const wcn_net_op& o) {
  return o.level_in >= 0 && o.level_out >= 0 && o.num_offsets > 0 && o.c_in > 0 && o.c_out > 0 && o.src >= 0 && o.dst >= 0 &&
         (o.kind == 1 || (o.kind == 0 && o.table >= 0));
}

}  // namespace

extern "C" int wcn_net_run(const wcn_net_op* ops, int32_t num_ops, const int64_t* rows, const wcn_net_buffer* buffers,
                           const wcn_net_table* tables, int dtype, int32_t* dev_status, void* stream) {
  if (!ops || num_ops < 0 || !rows || !buffers || !tables || (dtype != WCN_F16 && dtype != WCN_BF16)) return WCN_ERR_INVALID_PARAMETERS;
  // The first launch waits for everything before it (tables among it); the ones after it overlap with their
  // predecessors.
  struct Overlap {
    ~Overlap() { wcn_overlap_launches = false; }
  } until_return;
  for (int i = 0; i < num_ops; ++i) {
    const wcn_net_op& o = ops[i];
    if (!valid(o)) return WCN_ERR_INVALID_PARAMETERS;
    const int64_t n_in = rows[o.level_in], n_out = rows[o.level_out];
    if (n_out == 0) continue;
    const wcn_net_buffer &in = buffers[o.src], &out = buffers[o.dst];
    const void* src = at<const void*>(buffers, o.src, o.src_col);
    const void* res = at<const void*>(buffers, o.res, o.res_col);
    const int64_t res_ld = o.res >= 0 ? buffers[o.res].ld : 0;
    void* dst = at<void*>(buffers, o.dst, o.dst_col);
    int rc;
    if (o.kind == 1) {
      rc = wcn_conv_rows_fwd(src, n_in, in.ld, o.packed, o.table >= 0 ? tables[o.table].nbr : nullptr, n_out, o.num_offsets, o.c_in,
                             o.c_out_packed, o.c_out, dtype, o.scale, o.shift, res, res_ld, o.relu, dst, out.ld, dtype, dev_status,
                             stream);
    } else {
      rc = wcn_conv_fwd(WCN_CONV_AUTO, src, n_in, in.ld, o.weight, o.packed, tables[o.table].nbr, tables[o.table].out_rows, n_out,
                        o.num_offsets, o.c_in, o.c_out, dtype, o.scale, o.shift, res, res_ld, o.relu, dst, out.ld, dtype, 0,
                        nullptr, 0, dev_status, stream);
    }
    if (rc != WCN_OK) return rc;
    wcn_overlap_launches = true;
  }
  return WCN_OK;
}
