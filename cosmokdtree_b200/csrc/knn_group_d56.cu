// knn_group_d56.cu -- the kNN kernel with a group of lanes per query, d = 5 and 6.
#include "ckd_knn_group.cuh"

namespace ckd {
CKD_KNN_GROUP(5)
CKD_KNN_GROUP(6)
}  // namespace ckd
