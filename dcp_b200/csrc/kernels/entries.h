// C entries of the kernel library that other native code calls; the kernels' sources include this too, so the compiler
// compares the two.  All return 0, or a negative code when nothing ran.
#pragma once

// The levels of dQ of a backward call (see attn_levels.cuh), with that call's items, rows, heads and channels.  A null
// workspace: none.
struct DcpkDqLevels {
  const void* items;
  int n_items, n_levels, q_rows, hq, channels;
  void* workspace;      // dcpk_attn_bwd_workspace() bytes
};

extern "C" {
int dcpk_attn_fwd_pair(const void* q_arena, long q_rows, const void* kv_arena, long kv_rows, int hq, int hkv, const void* tiles,
                       int n_tiles, const void* kv_entries, int n_kv_entries, const void* masks, int n_mask_rows,
                       void* const* out_ptrs, float* const* lse_ptrs, int n_dst, int lse_stride_a, int lse_stride_b, int n_dst_a,
                       int out_type, int out_channels, float scale, int channels, const void* jobs, int n_jobs,
                       void* const* job_src_ptrs, void* const* job_dst_ptrs, int job_stat_stride, int* status, void* stream);
int dcpk_attn_bwd(const void* q_arena, const void* do_arena, long q_rows, const void* kv_arena, long kv_rows, int hq, int hkv,
                  const void* ctas, int n_ctas, const void* items, int n_items_total, int max_items, const void* masks,
                  int n_mask_rows, const float* lse, const float* delta, int stat_stride, float* const* dq_ptrs,
                  float* const* dkv_ptrs, int n_dst, float scale, int channels, int n_levels, void* workspace, int level_passes,
                  const void* jobs, int n_jobs, void* const* job_src_ptrs, void* const* job_dst_ptrs, int job_stat_stride, int* status,
                  void* stream);
long dcpk_attn_bwd_workspace(int n_items_total, long q_rows, int hq, int channels, int n_levels);
int dcpk_attn_bwd_parts(int n_ctas, int hkv, int group, int max_items, int n_items_total, int any_wave);
int dcpk_attn_bwd_prep(const void* o, const void* d_o, float* delta, int n_rows, int hq, int stat_stride, float* zero0, long nz0,
                       float* zero1, long nz1, const DcpkDqLevels* levels, void* stream);
int dcpk_attn_bwd_prep_cast(int type, const void* o, const void* d_o, int d, void* d_o_rows, float* delta, int n_rows, int hq,
                            int stat_stride, float* zero0, long nz0, float* zero1, long nz1, const DcpkDqLevels* levels, void* stream);
int dcpk_pad_cast_rows(int type, const void* src0, void* dst0, long rows0, const void* src1, void* dst1, long rows1, int d,
                       void* stream);
int dcpk_cut_cast_rows(int src_f32, int type, const void* src0, void* dst0, long rows0, const void* src1, void* dst1, long rows1,
                       int d, void* stream);
int dcpk_cut_cast_gradients(int type, const DcpkDqLevels* levels, const float* dq, void* gq, const float* dkv, void* gkv, long rows1, int d,
                            void* stream);
}
