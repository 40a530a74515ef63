// gw_math_tables.h -- generated by gen_math_tables.py; do not edit.
#pragma once
namespace gw {
namespace math64 {
constexpr unsigned long long kLog2e63 = 0xb8aa3b295c17f0bcull;  // 1/ln2, 63 fractional bits
constexpr unsigned long long kLn2 = 0xb17217f7d1cf79acull;      // ln2, 64 fractional bits
// 2048 times that, as two words
constexpr unsigned long long kLn2BiasHi = 0x58bull, kLn2BiasLo = 0x90bfbe8e7bcd6000ull;
constexpr unsigned long long kExp1 = 0xb17217f7d1cf79acull;  // ln2^1/1!, 64 fractional bits
constexpr unsigned long long kExp2 = 0x3d7f7bff058b1d51ull;  // ln2^2/2!, 64 fractional bits
constexpr unsigned long long kExp3 = 0xe35846b82505fc6ull;  // ln2^3/3!, 64 fractional bits
constexpr unsigned int kExp4 = 0x276556eu;  // ln2^4/4!, 32 fractional bits
constexpr unsigned int kExp5 = 0x576200u;  // ln2^5/5!, 32 fractional bits
constexpr unsigned long long kLog2 = 0x8000000000000000ull;  // 1/2, 64 fractional bits
constexpr unsigned long long kLog3 = 0x5555555555555555ull;  // 1/3, 64 fractional bits
constexpr unsigned int kLog4 = 0x40000000u;  // 1/4, 32 fractional bits
constexpr unsigned int kLog5 = 0x33333333u;  // 1/5, 32 fractional bits
constexpr unsigned int kLog6 = 0x2aaaaaabu;  // 1/6, 32 fractional bits
constexpr unsigned int kLog7 = 0x24924925u;  // 1/7, 32 fractional bits
// 2^(j/256), 63 fractional bits
#define GW_EXP2_TABLE \
    { \
        0x8000000000000000ull, 0x8058d7d2d5e5f6b1ull, 0x80b1ed4fd999ab6cull, 0x810b40a1d81406d4ull, \
        0x8164d1f3bc030773ull, 0x81bea1708dde6056ull, 0x8218af4373fc25ecull, 0x8272fb97b2a5894cull, \
        0x82cd8698ac2ba1d7ull, 0x83285071e0fc4547ull, 0x8383594eefb6ee37ull, 0x83dea15b9541b132ull, \
        0x843a28c3acde4046ull, 0x8495efb3303efd30ull, 0x84f1f656379c1a29ull, 0x854e3cd8f9c8c95dull, \
        0x85aac367cc487b15ull, 0x86078a2f23642a9full, 0x8664915b923fba04ull, 0x86c1d919caef5c88ull, \
        0x871f61969e8d1010ull, 0x877d2afefd4e256cull, 0x87db357ff698d792ull, 0x88398146b919f1d4ull, \
        0x88980e8092da8527ull, 0x88f6dd5af155ac6bull, 0x8955ee03618e5fddull, 0x89b540a7902557a4ull, \
        0x8a14d575496efd9aull, 0x8a74ac9a79896e47ull, 0x8ad4c6452c728924ull, 0x8b3522a38e1e1032ull, \
        0x8b95c1e3ea8bd6e7ull, 0x8bf6a434adde0085ull, 0x8c57c9c4646f4ddeull, 0x8cb932c1bae97a95ull, \
        0x8d1adf5b7e5ba9e6ull, 0x8d7ccfc09c50e2f8ull, 0x8ddf042022e69cd6ull, 0x8e417ca940e35a01ull, \
        0x8ea4398b45cd53c0ull, 0x8f073af5a2013520ull, 0x8f6a8117e6c8e5c4ull, 0x8fce0c21c6726481ull, \
        0x9031dc431466b1dcull, 0x9095f1abc540ca6bull, 0x90fa4c8beee4b12bull, 0x915eed13c89689d3ull, \
        0x91c3d373ab11c336ull, 0x9228ffdc10a051adull, 0x928e727d9531f9acull, 0x92f42b88f673aa7cull, \
        0x935a2b2f13e6e92cull, 0x93c071a0eef94bc1ull, 0x9426ff0fab1c04b6ull, 0x948dd3ac8ddb7ed3ull, \
        0x94f4efa8fef70961ull, 0x955c5336887894d5ull, 0x95c3fe86d6cc7fefull, 0x962bf1cbb8d97560ull, \
        0x96942d3720185a00ull, 0x96fcb0fb20ac4ba3ull, 0x97657d49f17ab08eull, 0x97ce9255ec4357abull, \
        0x9837f0518db8a96full, 0x98a1976f7597e996ull, 0x990b87e266c189aaull, 0x9975c1dd47518c77ull, \
        0x99e0459320b7fa65ull, 0x9a4b13371fd166caull, 0x9ab62afc94ff864aull, 0x9b218d16f441d63dull, \
        0x9b8d39b9d54e5539ull, 0x9bf93118f3aa4cc1ull, 0x9c6573682ec32c2dull, 0x9cd200db8a0774cbull, \
        0x9d3ed9a72cffb751ull, 0x9dabfdff6367a2aaull, 0x9e196e189d472420ull, 0x9e872a276f0b98ffull, \
        0x9ef5326091a111aeull, 0x9f6386f8e28ba651ull, 0x9fd228256400dd06ull, 0xa041161b3d0121beull, \
        0xa0b0510fb9714fc2ull, 0xa11fd9384a344cf7ull, 0xa18faeca8544b6e4ull, 0xa1ffd1fc25cea188ull, \
        0xa27043030c496819ull, 0xa2e102153e918f9eull, 0xa3520f68e802bb93ull, 0xa3c36b345991b47cull, \
        0xa43515ae09e6809eull, 0xa4a70f0c95768ec5ull, 0xa5195786be9ef339ull, 0xa58bef536dbeb6eeull, \
        0xa5fed6a9b15138eaull, 0xa6720dc0be08a20cull, 0xa6e594cfeee86b1eull, 0xa7596c0ec55ff55bull, \
        0xa7cd93b4e965356aull, 0xa8420bfa298f70d1ull, 0xa8b6d5167b320e09ull, 0xa92bef41fa77771bull, \
        0xa9a15ab4ea7c0ef8ull, 0xaa1717a7b5693979ull, 0xaa8d2652ec907629ull, 0xab0386ef48868de1ull, \
        0xab7a39b5a93ed337ull, 0xabf13edf162675e9ull, 0xac6896a4be3fe929ull, 0xace0413ff83e5d04ull, \
        0xad583eea42a14ac6ull, 0xadd08fdd43d01491ull, 0xae493452ca35b80eull, 0xaec22c84cc5c9465ull, \
        0xaf3b78ad690a4375ull, 0xafb51906e75b8661ull, 0xb02f0dcbb6e04584ull, 0xb0a957366fb7a3c9ull, \
        0xb123f581d2ac2590ull, 0xb19ee8e8c94feb09ull, 0xb21a31a66618fe3bull, 0xb295cff5e47db4a4ull, \
        0xb311c412a9112489ull, 0xb38e0e38419fae18ull, 0xb40aaea2654b9841ull, 0xb487a58cf4a9c180ull, \
        0xb504f333f9de6484ull, 0xb58297d3a8b9f0d2ull, 0xb60093a85ed5f76cull, 0xb67ee6eea3b22b8full, \
        0xb6fd91e328d17791ull, 0xb77c94c2c9d725e9ull, 0xb7fbefca8ca41e7cull, 0xb87ba337a1743834ull, \
        0xb8fbaf4762fb9ee9ull, 0xb97c143756844dbfull, 0xb9fcd2452c0b9debull, 0xba7de9aebe5fea09ull, \
        0xbaff5ab2133e45fbull, 0xbb81258d5b704b6full, 0xbc034a7ef2e9fb0dull, 0xbc85c9c560e7b269ull, \
        0xbd08a39f580c36bfull, 0xbd8bd84bb67ed483ull, 0xbe0f6809860993e2ull, 0xbe935317fc378238ull, \
        0xbf1799b67a731083ull, 0xbf9c3c248e2486f8ull, 0xc0213aa1f0d08db0ull, 0xc0a6956e8836ca8dull, \
        0xc12c4cca66709456ull, 0xc1b260f5ca0fbb33ull, 0xc238d2311e3d6673ull, 0xc2bfa0bcfad907c9ull, \
        0xc346ccda24976407ull, 0xc3ce56c98d21b15dull, 0xc4563ecc5334cb33ull, 0xc4de8523c2c07baaull, \
        0xc5672a115506daddull, 0xc5f02dd6b0bbc3d9ull, 0xc67990b5aa245f79ull, 0xc70352f04336c51eull, \
        0xc78d74c8abb9b15dull, 0xc817f681416452b2ull, 0xc8a2d85c8ffe2c45ull, 0xc92e1a9d517f0eccull, \
        0xc9b9bd866e2f27a3ull, 0xca45c15afcc72624ull, 0xcad2265e4290774eull, 0xcb5eecd3b38597c9ull, \
        0xcbec14fef2727c5dull, 0xcc799f23d11510e5ull, 0xcd078b86503dcdd2ull, 0xcd95da6a9ff06445ull, \
        0xce248c151f8480e4ull, 0xceb3a0ca5dc6a55dull, 0xcf4318cf191918c1ull, 0xcfd2f4683f94eeb5ull, \
        0xd06333daef2b2595ull, 0xd0f3d76c75c5db8dull, 0xd184df6251699ac6ull, 0xd2164c023056bcabull, \
        0xd2a81d91f12ae45aull, 0xd33a5457a3029054ull, 0xd3ccf099859ac379ull, 0xd45ff29e0972c561ull, \
        0xd4f35aabcfedfa1full, 0xd5872909ab75d18aull, 0xd61b5dfe9f9bce07ull, 0xd6aff9d1e13ba2feull, \
        0xd744fccad69d6af4ull, 0xd7da67311797f56aull, 0xd870394c6db32c84ull, 0xd9067364d44a929cull, \
        0xd99d15c278afd7b6ull, 0xda3420adba4d8704ull, 0xdacb946f2ac9cc72ull, 0xdb63714f8e295255ull, \
        0xdbfbb797daf23755ull, 0xdc9467913a4f1c92ull, 0xdd2d818508324c20ull, 0xddc705bcd378f7f0ull, \
        0xde60f4825e0e9124ull, 0xdefb4e1f9d1037f2ull, 0xdf9612deb8f04420ull, 0xe031430a0d99e627ull, \
        0xe0ccdeec2a94e111ull, 0xe168e6cfd3295d23ull, 0xe2055afffe83d369ull, 0xe2a23bc7d7d91226ull, \
        0xe33f8972be8a5a51ull, 0xe3dd444c46499619ull, 0xe47b6ca0373da88dull, 0xe51a02ba8e26d681ull, \
        0xe5b906e77c8348a8ull, 0xe658797368b3a717ull, 0xe6f85aaaee1fce22ull, 0xe798aadadd5b9cbfull, \
        0xe8396a503c4bdc68ull, 0xe8da9958464b42abull, 0xe97c38406c4f8c57ull, 0xea1e4756550eb27bull, \
        0xeac0c6e7dd24392full, 0xeb63b74317369840ull, 0xec0718b64c1cbddcull, 0xecaaeb8ffb03ab41ull, \
        0xed4f301ed9942b84ull, 0xedf3e6b1d418a491ull, 0xee990f980da3025bull, 0xef3eab20e032bc6bull, \
        0xefe4b99bdcdaf5cbull, 0xf08b3b58cbe8b76aull, 0xf13230a7ad094509ull, 0xf1d999d8b7708cc1ull, \
        0xf281773c59ffb13aull, 0xf329c9233b6bae9cull, 0xf3d28fde3a641a5bull, 0xf47bcbbe6db9fddfull, \
        0xf5257d152486cc2cull, 0xf5cfa433e6537290ull, 0xf67a416c733f846eull, 0xf7255510c4288239ull, \
        0xf7d0df730ad13bb9ull, 0xf87ce0e5b2094d9cull, 0xf92959bb5dd4ba74ull, 0xf9d64a46eb939f35ull, \
        0xfa83b2db722a033aull, 0xfb3193cc4227c3f4ull, 0xfbdfed6ce5f09c49ull, 0xfc8ec01121e447bbull, \
        0xfd3e0c0cf486c175ull, 0xfdedd1b496a89f35ull, 0xfe9e115c7b8f884cull, 0xff4ecb59511ec8a5ull, \
    }
// {c_j, -log(c_j / 2^16) with 64 fractional bits}
#define GW_LOG_TABLE \
    { \
        {65536ull, 0x0ull}, {65281ull, 0xff7f551588de02ull}, \
        {65028ull, 0x1fdfaa6b126788full}, {64777ull, 0x2fb6debf18dcec2ull}, \
        {64528ull, 0x3f7d51627807b25ull}, {64281ull, 0x4f32c10f02dd34dull}, \
        {64036ull, 0x5ed6ec2508c1368ull}, {63792ull, 0x6e7a009f8646364ull}, \
        {63551ull, 0x7dfaec4162c727full}, {63311ull, 0x8d7a5c4df4517ccull}, \
        {63073ull, 0x9ce79dd4f1085e8ull}, {62837ull, 0xac426d86b8a8dc0ull}, \
        {62602ull, 0xbb9b47b358e7559ull}, {62369ull, 0xcae148768667548ull}, \
        {62138ull, 0xda142b89080def2ull}, {61909ull, 0xe933ac58b121f92ull}, \
        {61681ull, 0xf8508600931532bull}, {61456ull, 0x1074883629640ad6ull}, \
        {61231ull, 0x1164e8eeaf5cde7eull}, {61009ull, 0x1252f32f8d183e9bull}, \
        {60788ull, 0x1340c796ac516a38ull}, {60568ull, 0x142e64bec266e772ull}, \
        {60350ull, 0x151ab33f13e03c65ull}, {60134ull, 0x1605aea96fc2aab5ull}, \
        {59919ull, 0x16f06a8afa8b45e3ull}, {59706ull, 0x17d9cc6db384b387ull}, \
        {59494ull, 0x18c2e9d642231d00ull}, {59284ull, 0x19aaa6464fbb998dull}, \
        {59075ull, 0x1a92193a589d6061ull}, {58868ull, 0x1b78242be5758a99ull}, \
        {58662ull, 0x1c5de08f760f3b25ull}, {58458ull, 0x1d422dd6d4051f7cull}, \
        {58255ull, 0x1e26276e8cf2acbfull}, {58053ull, 0x1f09cbc0254f2124ull}, \
        {57853ull, 0x1febf7320a3ca817ull}, {57654ull, 0x20cdc825a774d78bull}, \
        {57457ull, 0x21ae18fa06a47685ull}, {57261ull, 0x228e0a094f85827bull}, \
        {57066ull, 0x236d99aaa3d71e86ull}, {56872ull, 0x244cc63215d596e9ull}, \
        {56680ull, 0x252a65f047ea4543ull}, {56489ull, 0x26079d31c99025f7ull}, \
        {56300ull, 0x26e340407f3ec8c8ull}, {56112ull, 0x27be75626a0bed3bull}, \
        {55925ull, 0x28993ada3481c84eull}, {55739ull, 0x29738ee795cc124dull}, \
        {55554ull, 0x2a4d6fc753f06b50ull}, {55371ull, 0x2b25acb37c0d64c4ull}, \
        {55189ull, 0x2bfd70e1bfa76141ull}, {55008ull, 0x2cd4ba85475a6893ull}, \
        {54828ull, 0x2dab87ce60c4273eull}, {54649ull, 0x2e81d6ea81dbc97aull}, \
        {54472ull, 0x2f56720453b1fd62ull}, {54296ull, 0x302a8942fecf8819ull}, \
        {54121ull, 0x30fe1acaea639fe0ull}, {53947ull, 0x31d124bdc1ce76a0ull}, \
        {53774ull, 0x32a3a53a792d0292ull}, {53602ull, 0x33759a5d5218d791ull}, \
        {53431ull, 0x3447023fe09cbdd7ull}, {53262ull, 0x35169ff9d0ef940full}, \
        {53093ull, 0x35e6e69d3b47cbd0ull}, {52925ull, 0x36b69a3d1f93c8dcull}, \
        {52759ull, 0x37847ae884bb9c80ull}, {52594ull, 0x3851c2aba6931d29ull}, \
        {52429ull, 0x391faf8f3d344203ull}, {52266ull, 0x39ebc09c4bfd9f95ull}, \
        {52104ull, 0x3ab732d72ff6bc5dull}, {51942ull, 0x3b8347415cbafa1full}, \
        {51782ull, 0x3c4d76dc8305b9f7ull}, {51623ull, 0x3d1701a5d7b8e774ull}, \
        {51464ull, 0x3de12b97bd326c14ull}, {51307ull, 0x3ea967acd16ad3b8ull}, \
        {51151ull, 0x3f70f8db7a9bbaa1ull}, {50995ull, 0x40392616dafce571ull}, \
        {50841ull, 0x40ff5c5393d265f5ull}, {50687ull, 0x41c62c7f7560964bull}, \
        {50534ull, 0x428c4b89d8638b98ull}, {50383ull, 0x43506a5f36a1011dull}, \
        {50232ull, 0x44151fe749aaee08ull}, {50082ull, 0x44d91e0acca46e22ull}, \
        {49933ull, 0x459c62af3f17d1b4ull}, {49785ull, 0x465eebb823f5887dull}, \
        {49637ull, 0x47220905b639e83aull}, {49491ull, 0x47e315798c9409e0ull}, \
        {49345ull, 0x48a4b3ef4bad9385ull}, {49201ull, 0x49643b444c24b923ull}, \
        {49057ull, 0x4a245250110c2034ull}, {48914ull, 0x4ae3a2eb82361b7aull}, \
        {48771ull, 0x4ba382eb8494c270ull}, {48630ull, 0x4c614125741807aeull}, \
        {48490ull, 0x4d1e326b2efca65bull}, {48350ull, 0x4ddbaf8b6a532a9eull}, \
        {48211ull, 0x4e985d55fcdf76a6ull}, {48073ull, 0x4f5439978ce863afull}, \
        {47935ull, 0x5010a01a1ce18ec1ull}, {47799ull, 0x50cad3a87da88e80ull}, \
        {47663ull, 0x51858f08a37af51full}, {47528ull, 0x523f720137472b12ull}, \
        {47394ull, 0x52f87a5661ea2a08ull}, {47260ull, 0x53b208c98dd1a3baull}, \
        {47128ull, 0x5469561da9dfd653ull}, {46996ull, 0x5521270faed0a5c5ull}, \
        {46864ull, 0x55d97c5d2769acd2ull}, {46734ull, 0x568f88c477810a65ull}, \
        {46604ull, 0x574616fdc226f018ull}, {46475ull, 0x57fbbec3215376c4ull}, \
        {46346ull, 0x58b1e7cae9a65481ull}, {46219ull, 0x5965bccca9bfd92dull}, \
        {46092ull, 0x5a1a107afcd254b7ull}, {45965ull, 0x5acee388d6797625ull}, \
        {45840ull, 0x5b815aa910875506ull}, {45715ull, 0x5c344e8a280d3500ull}, \
        {45591ull, 0x5ce64fdb7fbfb419ull}, {45467ull, 0x5d98cd48fdcbb4c9ull}, \
        {45344ull, 0x5e4a557f7d1e889bull}, {45222ull, 0x5efae6290860eea4ull}, \
        {45101ull, 0x5faa7cef02462818ull}, {44980ull, 0x605a8c775059a9d9ull}, \
        {44859ull, 0x610b15687f0e5c82ull}, {44740ull, 0x61b92a6969b60ba6ull}, \
        {44621ull, 0x6267b61b9e28fb30ull}, {44502ull, 0x6316b92165a429d8ull}, \
        {44385ull, 0x63c3401d9a1c8082ull}, {44268ull, 0x64703bae0e2810a5ull}, \
        {44151ull, 0x651dac70b8e3d47aull}, {44035ull, 0x65ca160468edd914ull}, \
        {43920ull, 0x66757604c181f204ull}, {43805ull, 0x6721490b8346057full}, \
        {43691ull, 0x67cc0fb31e612520ull}, {43578ull, 0x6875c7941777b819ull}, \
        {43465ull, 0x691ff044298dc00full}, {43352ull, 0x69ca8a59af87a85aull}, \
        {43241ull, 0x6a728e6b0ea8a793ull}, {43130ull, 0x6b1b010a5784ae8eull}, \
        {43019ull, 0x6bc3e2c967638722ull}, {42909ull, 0x6c6bad3b486dc318ull}, \
        {42800ull, 0x6d125df0523c6a34ull}, {42691ull, 0x6db97b75def921f2ull}, \
        {42582ull, 0x6e61065a5ccbe970ull}, {42474ull, 0x6f07742c37162906ull}, \
        {42367ull, 0x6facc276b6b5e7eeull}, {42260ull, 0x70527bc457c89ab3ull}, \
        {42154ull, 0x70f7129f41fd3393ull}, {42049ull, 0x719a8490d8efa068ull}, \
        {41944ull, 0x723e5f1f8a6766b2ull}, {41839ull, 0x72e2a2d1970b6f8eull}, \
        {41735ull, 0x7385be2e95d15a95ull}, {41631ull, 0x742941b9d40e0e43ull}, \
        {41528ull, 0x74cb99f815af5107ull}, {41426ull, 0x756cc46c4bab71b5ull}, \
        {41324ull, 0x760e5496fadc45c7ull}, {41222ull, 0x76b04af8d697432eull}, \
        {41121ull, 0x775110133432711full}, {41021ull, 0x77f0a1652b124d0full}, \
        {40921ull, 0x7890966b20e1615dull}, {40821ull, 0x7930efa1fc245e27ull}, \
        {40722ull, 0x79d01187d23dd1faull}, {40623ull, 0x7a6f96966efc52a9ull}, \
        {40525ull, 0x7b0de1493d44f421ull}, {40428ull, 0x7baaef1a423e8175ull}, \
        {40330ull, 0x7c49fd7ec41bb178ull}, {40234ull, 0x7ce62cf3046a7dedull}, \
        {40137ull, 0x7d845de9c584b0e2ull}, {40042ull, 0x7e1faadd177bed2dull}, \
        {39946ull, 0x7ebcfa3df8ec75aeull}, {39851ull, 0x7f590583de3e4651ull}, \
        {39757ull, 0x7ff3ca21ce741cc5ull}, {39663ull, 0x808eec899a04906aull}, \
        {39569ull, 0x812a6d2d31a7f5e2ull}, {39476ull, 0x81c4a37e80e1d6deull}, \
        {39384ull, 0x825d8cee51b595b6ull}, {39291ull, 0x82f87ce935755ffbull}, \
        {39200ull, 0x839072e206f8e274ull}, {39108ull, 0x842a704274706af0ull}, \
        {39017ull, 0x84c31c7acaeb0190ull}, {38927ull, 0x855a74f739e665c7ull}, \
        {38837ull, 0x85f2272231d3183bull}, {38747ull, 0x868a33663a91fd02ull}, \
        {38658ull, 0x8720e82f85eb7a3dull}, {38569ull, 0x87b7f5e588e7e280ull}, \
        {38480ull, 0x884f5cf17264b69aull}, {38392ull, 0x88e568bc4d87be8dull}, \
        {38305ull, 0x897a16adb0aed884ull}, {38217ull, 0x8a10d229263aa70eull}, \
        {38131ull, 0x8aa4769905cdc99bull}, {38044ull, 0x8b3a295da2384e51ull}, \
        {37958ull, 0x8bce79df2354cfd6ull}, {37872ull, 0x8c63207fbaf82dc3ull}, \
        {37787ull, 0x8cf661a3961345edull}, {37702ull, 0x8d89f7ac2836dcb4ull}, \
        {37618ull, 0x8e1c24fcd567c232ull}, {37533ull, 0x8eb064f33de4980bull}, \
        {37450ull, 0x8f417af4a20561f1ull}, {37366ull, 0x8fd4a45c537c5805ull}, \
        {37283ull, 0x9066608cb86d605eull}, {37201ull, 0x90f6ace49f8a3c67ull}, \
        {37118ull, 0x91890ebe121a0b4dull}, {37036ull, 0x9219ff7a52519b1bull}, \
        {36955ull, 0x92a97c75bc7f783eull}, {36874ull, 0x93394a0b34172277ull}, \
        {36793ull, 0x93c9689579a7a4fcull}, {36712ull, 0x9459d86fe75bfd5aull}, \
        {36632ull, 0x94e8cff686040ff3ull}, {36552ull, 0x957817815f255709ull}, \
        {36473ull, 0x9605e36b273b687full}, {36394ull, 0x9693fe0acc2579e6ull}, \
        {36315ull, 0x972267b7e0a4a48cull}, {36236ull, 0x97b120ca89f230b5ull}, \
        {36158ull, 0x983e599a8a85ec7eull}, {36081ull, 0x98ca0f7ec9b20486ull}, \
        {36003ull, 0x9957e3c8d19d6ae7ull}, {35926ull, 0x99e433d1f80e6b8bull}, \
        {35849ull, 0x9a70d0ed015690c7ull}, {35773ull, 0x9afbe66f64b4d7d7ull}, \
        {35697ull, 0x9b8747ab4b6ea41bull}, {35621ull, 0x9c12f4f357800c36ull}, \
        {35545ull, 0x9c9eee9ab270cd3cull}, {35470ull, 0x9d295bf40731c82bull}, \
        {35395ull, 0x9db4145000431579ull}, {35321ull, 0x9e3d3d003c9455e3ull}, \
        {35247ull, 0x9ec6af54823eefa6ull}, {35173ull, 0x9f506b9c0f2acbd0ull}, \
        {35099ull, 0x9fda7226a16c0cccull}, {35026ull, 0xa062e44475890483ull}, \
        {34953ull, 0xa0eb9f42959539f9ull}, {34880ull, 0xa174a36f0405f810ull}, \
        {34808ull, 0xa1fc0f183ef2f584ull}, {34736ull, 0xa283c28a2e57ec28ull}, \
        {34664ull, 0xa30bbe1114f5ff13ull}, {34593ull, 0xa3921cfac4e0be29ull}, \
        {34522ull, 0xa418c2910eccd714ull}, {34451ull, 0xa49faf1e720b4054ull}, \
        {34380ull, 0xa526e2ede3f59ee7ull}, {34310ull, 0xa5ac754bc844925bull}, \
        {34240ull, 0xa6324d7f8770ad8dull}, {34170ull, 0xa6b86bd24de9aee1ull}, \
        {34101ull, 0xa73ce48f7563605bull}, {34031ull, 0xa7c38efa89fbc2a7ull}, \
        {33962ull, 0xa84892600b8b5a5cull}, {33894ull, 0xa8cbec06923395c0ull}, \
        {33826ull, 0xa94f8934a02b24f7ull}, {33757ull, 0xa9d55b2dcd306552ull}, \
        {33690ull, 0xaa578f3e0b6b6de8ull}, {33622ull, 0xaadbf8a5d3a05444ull}, \
        {33555ull, 0xab5eb2ae3d245587ull}, {33488ull, 0xabe1af9a480c1dd3ull}, \
        {33421ull, 0xac64efae8ace3f58ull}, {33355ull, 0xace67c30c5279785ull}, \
        {33289ull, 0xad684a632717b697ull}, {33223ull, 0xadea5a886fd2d5cbull}, \
        {33157ull, 0xae6cace3c47ce9b2ull}, {33092ull, 0xaeed46ba0a8f8cf5ull}, \
        {33027ull, 0xaf6e214b08f92fc2ull}, {32962ull, 0xafef3cd809d90d39ull}, \
        {32897ull, 0xb07099a2ba4872fbull}, {32833ull, 0xb0f038eea961ee78ull}, \
    }
}  // namespace math64
}  // namespace gw
